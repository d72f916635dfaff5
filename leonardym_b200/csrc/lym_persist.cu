// CG on A = Q Q + sigma (Q = gamma5 D of the Wilson or Wilson-clover operator, FP64, both
// parities) in one cooperative launch, for lattices whose blocks all fit on the GPU at once.
//
// On a small lattice an iteration is latency: three launches (lym_split.cu: q = Q p with <p, A p>,
// A p with x, r and |r|^2, the direction) each pay a launch, the state's gate, the links' and
// clover words' trip from L2 and the last block's sum.  Here every block keeps its 32 sites for the
// whole solve: x, r, p in registers and shared memory, its clover words in shared memory, its links
// in L1, and an iteration is two phases with a grid barrier after each:
//   1. p_k = r + beta p_{k-1}, formed at the neighbours as it is read; q = Q p_k; <p_k, A p_k>;
//   2. A p_k = Q q + sigma p_k; x += alpha p_k, r -= alpha A p_k; |r|^2.
// The sums are per-block partial sums that every block adds up itself, in a fixed order, after the
// barrier, and then runs the CG step's scalars (OpCGUpdate) on its own copy: all copies agree bit
// for bit.  Directions alternate between two buffers and partial sums between two
// halves, so that nobody overwrites what a slower block may still read.
// 8^4 clover, 106 iterations: 1.04 ms (9.8 us an iteration) against 2.2 ms; whole solve with its
// transfers 1.14 against 2.37 ms.
#include "lym_blas.cuh"
#include "lym_internal.h"
#include "lym_solver_ops.cuh"
#include "lym_split.cuh"

namespace lym {

namespace {

using namespace split;

template <class GaugeT> struct PersistArg {
    Geom g;
    GaugeT U;
    const double2 *clover;
    double b, sigma;
    SpinorD x, r, q, p[2];  // full spinors; p[k & 1] holds p_k
    CGState *state;
    double *partials;       // 2 * gridDim.x
    unsigned int *arrived;  // zero at the launch
    int *err;               // set to 1 when a barrier wait gave up
    int steps;              // iterations of this launch at most
};

LYM_D C load_cg(const SpinorD &v, int word, int h)  // from L2: other SMs write these vectors
{
    const double2 w = __ldcg(v.v + (size_t)word * v.stride + h);
    return C{w.x, w.y};
}

// Grid barrier of a cooperative launch (all blocks resident).  The wait is bounded, about a
// second; false when it ran out.  target: arrivals expected so far.
LYM_D bool grid_barrier(unsigned int *arrived, unsigned int target, bool *ok)
{
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        atomicAdd(arrived, 1u);
        bool done = false;
        for (int i = 0; i < (1 << 21); ++i) {
            unsigned int v;
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];\n" : "=r"(v) : "l"(arrived) : "memory");
            if (v >= target) {
                done = true;
                break;
            }
        }
        __threadfence();
        *ok = done;
    }
    __syncthreads();
    return *ok;
}

template <int MINB, class GaugeT>
__global__ void __launch_bounds__(kSplitThreads, MINB) cg_persist_kernel(const PersistArg<GaugeT> a)
{
    extern __shared__ __align__(16) double2 smem[];
    double2 *const fetch = smem + threadIdx.x;                    // clover words
    double2 *const own_x = fetch + kCloverWords * kSplitThreads;  // x, 3 words a thread
    __shared__ double wsum[2][kSplitThreads / 32];
    __shared__ bool ok;
    const Geom &g = a.g;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int d = (lane >> 3) & 1, k = lane >> 4, p = warp >> 1;
    const int hr = blockIdx.x * (kSplitSites / 2) + (warp & 1) * 8 + (lane & 7);
    const bool in = hr < g.Vh;
    const int h = in ? hr : g.Vh - 1;
    int c[4];
    site_coords(g, h, p, c);
    const int s = lex_of(g, c[0], c[1], c[2], c[3]);
    const int sp = 3 * (2 * d + k);
    const SpinorD xv = a.x.par(p), rv = a.r.par(p), qv = a.q.par(p);
    const SpinorD rn = a.r.par(1 - p), qn = a.q.par(1 - p);
    if (a.clover) fetch_clover(fetch, a.clover, g.stride, p, h, k, d);
    // every thread's copy of the scalars
    const CGState st = *a.state;
    int it = st.iter;
    double rr = st.rr, rr_prev = st.rr_prev, rr_max = st.rr_max, alpha = st.alpha.x, beta = st.beta;
    int flags = 0;  // 1 pause, 2 converged, 4 failed
    C r[3], pk[3];
    const SpinorD last = a.p[(it + 1) & 1].par(p);
#pragma unroll
    for (int m = 0; m < 3; ++m) {
        own_x[m * kSplitThreads] = xv.v[(size_t)(sp + m) * xv.stride + h];
        r[m] = load_cg(rv, sp + m, h);
        pk[m] = beta != 0.0 ? load_cg(last, sp + m, h) : C{0.0, 0.0};
    }
    asm volatile("cp.async.wait_all;\n" ::: "memory");
    auto put = [&](const SpinorD &v, int m, C z) {
        if (in) v.v[(size_t)(sp + m) * v.stride + h] = make_double2(z.re, z.im);
    };
    // rows of Q v from the hopping term and the own-site vector
    auto finish = [&](const C acc[3], const C own[3], C res[3]) {
        if (a.clover) {
            C oth[3];
#pragma unroll
            for (int m = 0; m < 3; ++m) oth[m] = shfl_xor(own[m], 16);
            clover_rows([&](int w) { return fetch[w * kSplitThreads]; }, k, own, oth, res);
        } else {
#pragma unroll
            for (int m = 0; m < 3; ++m) res[m] = own[m];
        }
#pragma unroll
        for (int m = 0; m < 3; ++m) {
            fma_r(res[m], a.b, acc[m]);
            if (d) res[m] = -res[m];
        }
    };
    // the block's sum of v, in every thread; slot: 0 and 1 in turn
    auto block_total = [&](double v, int slot) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
        if (lane == 0) wsum[slot][warp] = v;
        __syncthreads();
        return (wsum[slot][0] + wsum[slot][1]) + (wsum[slot][2] + wsum[slot][3]);
    };
    unsigned int target = 0;
    // the block's part of a sum, then the barrier; false when it gave up
    auto contribute = [&](double v, int half) {
        const double t = block_total(in ? v : 0.0, 0);
        if (threadIdx.x == 0) a.partials[(size_t)half * gridDim.x + blockIdx.x] = t;
        target += gridDim.x;
        return grid_barrier(a.arrived, target, &ok);
    };
    // this thread's share of the blocks' parts (their sum over the block is the grid's)
    auto collect = [&](int half) {
        double u = 0.0;
        for (int i = threadIdx.x; i < (int)gridDim.x; i += kSplitThreads)
            u += __ldcg(a.partials + (size_t)half * gridDim.x + i);
        return u;
    };
    bool good = true;
    for (int n = 0; n < a.steps && !(flags & 1); ++n) {
        const SpinorD pnew = a.p[it & 1].par(p), pold = a.p[(it + 1) & 1].par(1 - p);
        C acc[3], q[3], ap[3];
#pragma unroll
        for (int m = 0; m < 3; ++m) {
            const C z = pk[m];
            pk[m] = r[m];
            if (beta != 0.0) fma_r(pk[m], beta, z);
            put(pnew, m, pk[m]);
        }
        if (beta != 0.0)
            split_hopping(g, [&](int w, int sn) {
                C z = load_cg(rn, w, sn >> 1);
                fma_r(z, beta, load_cg(pold, w, sn >> 1));
                return z;
            }, a.U, p, h, s, c, k, d, acc);
        else
            split_hopping(g, [&](int w, int sn) { return load_cg(rn, w, sn >> 1); }, a.U, p, h, s, c, k, d, acc);
        finish(acc, pk, q);
        double part = 0.0, pp = 0.0;
#pragma unroll
        for (int m = 0; m < 3; ++m) {
            put(qv, m, q[m]);
            part += q[m].re * q[m].re + q[m].im * q[m].im;
            pp += pk[m].re * pk[m].re + pk[m].im * pk[m].im;
        }
        if (a.sigma != 0.0) part += a.sigma * pp;
        if (!(good = contribute(part, 0))) break;
        const double pap = collect(0);  // needed only after the stencil
        split_hopping(g, [&](int w, int sn) { return load_cg(qn, w, sn >> 1); }, a.U, p, h, s, c, k, d, acc);
        finish(acc, q, ap);
        alpha = rr / block_total(pap, 1);
        part = 0.0;
#pragma unroll
        for (int m = 0; m < 3; ++m) {
            fma_r(ap[m], a.sigma, pk[m]);
            double2 &x = own_x[m * kSplitThreads];
            x.x = fma(alpha, pk[m].re, x.x);
            x.y = fma(alpha, pk[m].im, x.y);
            fma_r(r[m], -alpha, ap[m]);
            part += r[m].re * r[m].re + r[m].im * r[m].im;
            put(rv, m, r[m]);
        }
        if (!(good = contribute(part, 1))) break;
        // the scalars of OpCGUpdate (no reliable updates in FP64)
        const double rr_new = block_total(collect(1), 1);
        ++it;
        rr_prev = rr;
        beta = rr_new / rr;
        rr = rr_new;
        rr_max = fmax(rr_max, rr);
        if (!(rr == rr)) flags = 1 | 4;
        else if (rr < st.eps) flags = 1 | 2;
        else if (it >= st.max_iter) flags = 1;
    }
#pragma unroll
    for (int m = 0; m < 3; ++m) {
        const double2 x = own_x[m * kSplitThreads];
        put(xv, m, C{x.x, x.y});
    }
    if (threadIdx.x == 0) {
        if (!good) atomicOr(a.err, 1);
        if (blockIdx.x == 0) {
            CGState out = st;
            out.iter = it;
            out.rr = rr;
            out.rr_prev = rr_prev;
            out.rr_max = rr_max;
            out.alpha = make_double2(alpha, 0.0);
            out.beta = beta;
            out.pause = flags & 1;
            out.converged = out.need_update = (flags >> 1) & 1;
            out.failed = (flags >> 2) & 1;
            *a.state = out;
        }
    }
}

constexpr int kPersistSmem = (kCloverWords + 3) * kSplitThreads * 16;

int persist_blocks(const Geom &g) { return (g.Vh + kSplitSites / 2 - 1) / (kSplitSites / 2); }

// Blocks per SM the kernel is compiled for: 2 (all the registers it wants) where that holds the
// lattice, else 4.  0: it does not fit, or the GPU has no cooperative launch.
template <class GaugeT> int residency(const Geom &g, int device)
{
    int sms = 0, coop = 0;
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device) != cudaSuccess ||
        cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, device) != cudaSuccess || !coop)
        return 0;
    auto holds = [&](const void *kernel) {
        int per = 0;
        return cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kernel, kSplitThreads, kPersistSmem) == cudaSuccess &&
               persist_blocks(g) <= sms * per;
    };
    if (holds((const void *)cg_persist_kernel<2, GaugeT>)) return 2;
    return holds((const void *)cg_persist_kernel<4, GaugeT>) ? 4 : 0;
}

template <class GaugeT>
cudaError_t run(const DslashParams &P, int minb, const Spinor &p0, const Spinor &p1, const Spinor &x, const Spinor &r,
                const Spinor &q, CGState *state, double *partials, unsigned int *arrived, int *err, int steps,
                const GaugeT &U, cudaStream_t st)
{
    PersistArg<GaugeT> a{P.g,     U,       (const double2 *)P.clover, P.b,   P.sigma, x.d(), r.d(), q.d(), {p0.d(), p1.d()},
                         state, partials, arrived,                   err, steps};
    const cudaError_t e = cudaMemsetAsync(arrived, 0, sizeof(unsigned int), st);
    if (e != cudaSuccess) return e;
    void *args[] = {&a};
    const void *kernel = minb == 2 ? (const void *)cg_persist_kernel<2, GaugeT> : (const void *)cg_persist_kernel<4, GaugeT>;
    return cudaLaunchCooperativeKernel(kernel, dim3(persist_blocks(P.g)), dim3(kSplitThreads), args, kPersistSmem, st);
}

}  // namespace

int cg_persist_residency(const Geom &g, int rep, int device)
{
    return rep == REP_SU3 ? residency<GaugeD18>(g, device) : residency<GaugeD9>(g, device);
}
int cg_persist_partials(const Geom &g) { return 2 * persist_blocks(g); }

cudaError_t launch_cg_persist(const DslashParams &P, int minb, const Spinor &p0, const Spinor &p1, const Spinor &x,
                              const Spinor &r, const Spinor &q, void *state, double *partials, unsigned int *arrived,
                              int *err, int steps, cudaStream_t st)
{
    const int s = P.g.stride;
    CGState *cs = (CGState *)state;
    if (P.rep == REP_SU3)
        return run(P, minb, p0, p1, x, r, q, cs, partials, arrived, err, steps, GaugeD18{(const double2 *)P.U->d64, s}, st);
    return run(P, minb, p0, p1, x, r, q, cs, partials, arrived, err, steps, GaugeD9{(const double *)P.U->d64, s}, st);
}

}  // namespace lym
