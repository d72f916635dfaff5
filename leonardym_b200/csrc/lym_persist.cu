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
//
// ms a solve to 1e-10 (SquareImproved, kappa 0.12, 106 to 120 iterations), in one launch and with
// launches per iteration (after a launch made to give up at once, about 0.1 ms): 8^4 1.17 and 2.80, 8^3 x 18 1.62 and 3.36; with 4 blocks per SM 8^3 x 20
// 2.01 and 3.57, 6 x 8 x 14 x 28 2.63 and 4.21.  8^4 is 9.9 us an iteration: two barriers and two
// chains of L2 loads.
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
    BarrierWait wait;
    int steps;              // iterations of this launch at most
};

LYM_D C load_cg(const SpinorD &v, int word, int h)  // from L2: other SMs write these vectors
{
    const double2 w = __ldcg(v.v + (size_t)word * v.stride + h);
    return C{w.x, w.y};
}

// Grid barrier of a cooperative launch (all blocks resident) in two halves, work that needs no other
// block's results between them.
LYM_D void grid_arrive(unsigned int *arrived)
{
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        atomicAdd(arrived, 1u);
    }
}
// target: arrivals expected so far.  The wait is bounded; false when it ran out.
LYM_D bool grid_wait(unsigned int *arrived, unsigned int target, int polls, bool *ok)
{
    if (threadIdx.x == 0) {
        bool done = false;
        for (int i = 0; i < polls; ++i) {
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
LYM_D bool grid_barrier(unsigned int *arrived, unsigned int target, int polls, bool *ok)
{
    grid_arrive(arrived);
    return grid_wait(arrived, target, polls, ok);
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
    unsigned int target = a.wait.extra;
    // the block's part of a sum, then the barrier; false when it gave up
    auto contribute = [&](double v, int half) {
        const double t = block_total(in ? v : 0.0, 0);
        if (threadIdx.x == 0) a.partials[(size_t)half * gridDim.x + blockIdx.x] = t;
        target += gridDim.x;
        return grid_barrier(a.arrived, target, a.wait.polls, &ok);
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
        if (!good) {  // the host starts the solve again with launches per iteration
            atomicOr(a.err, 1);
        } else if (blockIdx.x == 0) {
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
                const Spinor &q, CGState *state, double *partials, unsigned int *arrived, int *err, BarrierWait wait,
                int steps, const GaugeT &U, cudaStream_t st)
{
    PersistArg<GaugeT> a{P.g,   U,     (const double2 *)P.clover, P.b,     P.sigma, x.d(), r.d(), q.d(), {p0.d(), p1.d()},
                         state, partials, arrived,                   err,     wait,    steps};
    const cudaError_t e = cudaMemsetAsync(arrived, 0, sizeof(unsigned int), st);
    if (e != cudaSuccess) return e;
    void *args[] = {&a};
    const void *kernel = minb == 2 ? (const void *)cg_persist_kernel<2, GaugeT> : (const void *)cg_persist_kernel<4, GaugeT>;
    return cudaLaunchCooperativeKernel(kernel, dim3(persist_blocks(P.g)), dim3(kSplitThreads), args, kPersistSmem, st);
}

// ------------------------------------------------------------- multishift --
// The FP64 multishift CG (multishift_cg: windowed shifted updates from a ring of residuals) on
// Q Q + shifts in one cooperative launch.  Every block walks its tiles of 32 half-sites in each
// phase; the vectors stay in L2 and the MultishiftState is replicated in every block's shared
// memory.  EO: Q = gamma5 S on the odd sites, A = 1 + sigma on the even ones, whose tiles come last.
// A step: [EO: tmp = T^-1 H p;] q = Q p with <p, A p>; [tmp = T^-1 H q;] r_{k+1} = r_k - alpha A p
// with |r_{k+1}|^2, a grid barrier after each; p_k = r_k + beta p_{k-1} is formed where it is read,
// as in the CG above.  The shifts' scalars and, after kMsWin steps or the last, the window's updates
// of x_i and P_i run while a block waits for the others.
// Latency bound (a stencil phase 7 us with 128 registers a thread; polling without the acquire,
// reads through L1 and links fetched into shared memory while waiting change nothing at the larger
// size).  8 shifts to 1e-10, ms a solve in one launch and with launches per step as above: even-odd, kappa
// 0.1365, 8^4 3.6 and 4.8, 10 x 12 x 14 x 18 9.4 and 11.5; SquareImproved, kappa 0.13, 8^4 3.6 and
// 6.2, 10 x 12 x 14 x 18 10.6 and 14.9.
template <class GaugeT> struct PersistMsArg {
    Geom g;
    GaugeT U;
    const double2 *T, *Ti;   // null without clover
    double b, sigma;
    const SpinorD *ring, *x, *dir;  // device arrays: kMsWin + 1 residuals, solutions, window directions
    SpinorD p[2], q;                // full spinors; p[k & 1] holds p_k
    SpinorD tmp;                    // EO: an even half spinor
    MultishiftState *state;
    double *partials;               // 2 * gridDim.x
    unsigned int *arrived;
    int *err;
    BarrierWait wait;
    int nshift, steps;
};

template <bool EO, class GaugeT>
__global__ void __launch_bounds__(kSplitThreads, 4) ms_persist_kernel(const PersistMsArg<GaugeT> a)
{
    __shared__ __align__(16) MultishiftState st;
    __shared__ SpinorD ring[kMsWin + 1];
    __shared__ double wsum[2][kSplitThreads / 32];
    __shared__ bool ok;
    const Geom &g = a.g;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int d = (lane >> 3) & 1, k = lane >> 4;
    const int sp = 3 * (2 * d + k);
    const int tiles = (g.Vh + kSplitSites - 1) / kSplitSites;
    static_assert(sizeof(MultishiftState) % sizeof(int) == 0, "copied by words");
    for (int i = threadIdx.x; i < (int)(sizeof(st) / sizeof(int)); i += kSplitThreads)
        reinterpret_cast<int *>(&st)[i] = reinterpret_cast<const int *>(a.state)[i];
    if (threadIdx.x <= kMsWin) ring[threadIdx.x] = a.ring[threadIdx.x];
    __syncthreads();
    auto block_total = [&](double v, int slot) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
        if (lane == 0) wsum[slot][warp] = v;
        __syncthreads();
        return (wsum[slot][0] + wsum[slot][1]) + (wsum[slot][2] + wsum[slot][3]);
    };
    unsigned int target = a.wait.extra;
    auto arrive = [&]() {
        target += gridDim.x;
        grid_arrive(a.arrived);
    };
    auto wait = [&]() { return grid_wait(a.arrived, target, a.wait.polls, &ok); };
    // the block's part of a sum, then the barrier's first half
    auto contribute = [&](double v, int half) {
        const double t = block_total(v, 0);
        if (threadIdx.x == 0) a.partials[(size_t)half * gridDim.x + blockIdx.x] = t;
        arrive();
    };
    // this thread's share of the blocks' parts
    auto collect = [&](int half) {
        double u = 0.0;
        for (int i = threadIdx.x; i < (int)gridDim.x; i += kSplitThreads)
            u += __ldcg(a.partials + (size_t)half * gridDim.x + i);
        return u;
    };
    struct At {
        bool in;
        int p, h, s, c[4];
    };
    auto place = [&](int tile, int p) {
        At t;
        const int hr = tile * kSplitSites + warp * 8 + (lane & 7);
        t.in = hr < g.Vh;
        t.p = p;
        t.h = t.in ? hr : g.Vh - 1;
        site_coords(g, t.h, p, t.c);
        t.s = lex_of(g, t.c[0], t.c[1], t.c[2], t.c[3]);
        return t;
    };
    // the tiles of both parities: EO the odd ones, which have the stencil, first
    auto item = [&](int i) { return EO ? (i < tiles ? place(i, 1) : place(i - tiles, 0)) : place(i >> 1, i & 1); };
    auto put = [&](const SpinorD &v, const At &t, int m, C z) {
        if (t.in) v.v[(size_t)(sp + m) * v.stride + t.h] = make_double2(z.re, z.im);
    };
    auto rows = [&](const double2 *clover, const At &t, const C own[3], C res[3]) {
        C oth[3];
#pragma unroll
        for (int m = 0; m < 3; ++m) oth[m] = shfl_xor(own[m], 16);
        const double2 *const base = clover + (size_t)((t.p * 2 + d) * 18) * g.stride + t.h;
        clover_rows([&](int w) { return __ldg(base + (size_t)clover_word(w, k) * g.stride); }, k, own, oth, res);
    };
    // EO: tmp = T^-1 H v on the even sites, load(w, sn) the words of v
    auto even_half = [&](auto load) {
        for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
            const At t = place(tile, 0);
            C acc[3], res[3];
            split_hopping(g, load, a.U, 0, t.h, t.s, t.c, k, d, acc);
            if (a.Ti) rows(a.Ti, t, acc, res);
#pragma unroll
            for (int m = 0; m < 3; ++m) put(a.tmp, t, m, a.Ti ? res[m] : acc[m]);
        }
    };
    // rows of Q v at a site: own-site words and the hopping term's input
    auto product = [&](auto load, const At &t, const C own[3], C res[3]) {
        C acc[3];
        split_hopping(g, load, a.U, t.p, t.h, t.s, t.c, k, d, acc);
        if (a.T) {
            rows(a.T, t, own, res);
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
    int it = st.iter;
    double rr = st.rr, beta = st.beta;
    const bool stopped = st.stop != 0;
    bool pending = false;  // the scalars of the residual rr have not been stepped yet
    // the shifts' scalars after a residual; the window's updates (ms_flush_kernel) when it is full
    auto settle = [&]() {
        pending = false;
        ms_residual_step(&st, rr);
        __syncthreads();
        if (st.win < kMsWin && !st.stop) return;
        const int m = st.win, k0 = ms_window_start(&st), words = 2 * 12 * g.stride;
        for (int o = blockIdx.x * kSplitThreads + threadIdx.x; m > 0 && o < words; o += gridDim.x * kSplitThreads) {
            double2 R[kMsWin];
#pragma unroll
            for (int j = 0; j < kMsWin; ++j)
                if (j < m) R[j] = __ldcg(ring[(k0 + 1 + j) % (kMsWin + 1)].v + o);
            for (int i = 0; i < a.nshift; ++i) {
                if (!st.xupd[i]) continue;
                double2 *const xp = a.x[i].v + o, *const pp = a.dir[i].v + o;
                const double2 P = *pp;
                double2 X = *xp, Q = word_scale(st.cp[i][0], P);
                word_add(X, st.cx[i][0], P);
#pragma unroll
                for (int j = 0; j < kMsWin; ++j)
                    if (j < m) {
                        if (j < m - 1) word_add(X, st.cx[i][j + 1], R[j]);  // the last one is not in x yet
                        word_add(Q, st.cp[i][j + 1], R[j]);
                    }
                *xp = X;
                if (st.pupd[i] && st.active[i] == 1) *pp = Q;
            }
        }
        __syncthreads();
        if ((int)threadIdx.x < a.nshift) {
            const int i = threadIdx.x;
            st.xupd[i] = st.pupd[i] = 0;
            for (int j = 0; j <= kMsWin; ++j) st.cx[i][j] = st.cp[i][j] = 0.0;
            st.cp[i][0] = 1.0;
        }
        if (threadIdx.x == 0) st.win = 0;
        __syncthreads();
    };
    bool good = true;
    for (int n = 0; n < a.steps && !stopped; ++n) {
        const SpinorD r = ring[it % (kMsWin + 1)], rnext = ring[(it + 1) % (kMsWin + 1)];
        const SpinorD pnew = a.p[it & 1], pold = a.p[(it + 1) & 1];
        auto direction = [&](int p, int w, int h) {  // word w of p_k
            C z = load_cg(r.par(p), w, h);
            if (beta != 0.0) fma_r(z, beta, load_cg(pold.par(p), w, h));
            return z;
        };
        const SpinorD tmp = a.tmp;
        auto load_tmp = [&](int w, int sn) { return load_cg(tmp, w, sn >> 1); };
        if (EO) {
            even_half([&](int w, int sn) { return direction(1, w, sn >> 1); });
            arrive();
            if (pending) settle();
            if (!(good = wait()) || st.stop) break;
        }
        double part = 0.0;
        for (int i = blockIdx.x; i < 2 * tiles; i += gridDim.x) {
            const At t = item(i);
            C own[3], res[3];
            double pp = 0.0, qq = 0.0;
#pragma unroll
            for (int m = 0; m < 3; ++m) {
                own[m] = direction(t.p, sp + m, t.h);
                put(pnew.par(t.p), t, m, own[m]);
                pp += own[m].re * own[m].re + own[m].im * own[m].im;
            }
            if (EO && t.p == 0) {
                qq = pp;
            } else {
                if (EO) product(load_tmp, t, own, res);
                else product([&](int w, int sn) { return direction(1 - t.p, w, sn >> 1); }, t, own, res);
#pragma unroll
                for (int m = 0; m < 3; ++m) {
                    put(a.q.par(t.p), t, m, res[m]);
                    qq += res[m].re * res[m].re + res[m].im * res[m].im;
                }
            }
            if (t.in) part += qq + a.sigma * pp;
        }
        contribute(part, 0);
        if (!EO && pending) settle();
        if (!(good = wait()) || st.stop) break;
        const double share = collect(0);
        if (EO) {
            const SpinorD q1 = a.q.par(1);
            even_half([&](int w, int sn) { return load_cg(q1, w, sn >> 1); });
            arrive();
        }
        const double pap = block_total(share, 1), alpha = rr / pap;
        if (EO && !(good = wait())) break;
        part = 0.0;
        for (int i = blockIdx.x; i < 2 * tiles; i += gridDim.x) {
            const At t = item(i);
            const SpinorD qv = a.q.par(t.p), qn = a.q.par(1 - t.p);
            C own[3], ap[3];
            if (!(EO && t.p == 0)) {
#pragma unroll
                for (int m = 0; m < 3; ++m) own[m] = load_cg(qv, sp + m, t.h);
                if (EO) product(load_tmp, t, own, ap);
                else product([&](int w, int sn) { return load_cg(qn, w, sn >> 1); }, t, own, ap);
            }
            double nrm = 0.0;
#pragma unroll
            for (int m = 0; m < 3; ++m) {
                const C pv = load_cg(pnew.par(t.p), sp + m, t.h);
                if (EO && t.p == 0) ap[m] = pv;
                fma_r(ap[m], a.sigma, pv);
                C rv = load_cg(r.par(t.p), sp + m, t.h);
                fma_r(rv, -alpha, ap[m]);
                nrm += rv.re * rv.re + rv.im * rv.im;
                put(rnext.par(t.p), t, m, rv);
            }
            if (t.in) part += nrm;
        }
        contribute(part, 1);
        ms_alpha_step(&st, pap);
        if (!(good = wait())) break;
        const double rr_new = block_total(collect(1), 1);
        beta = rr_new / rr;
        rr = rr_new;
        ++it;
        pending = true;
    }
    __syncthreads();
    if (good && pending) settle();
    if (threadIdx.x == 0 && !good) atomicOr(a.err, 1);
    if (blockIdx.x == 0 && good)
        for (int i = threadIdx.x; i < (int)(sizeof(st) / sizeof(int)); i += kSplitThreads)
            reinterpret_cast<int *>(a.state)[i] = reinterpret_cast<const int *>(&st)[i];
}

template <bool EO, class GaugeT>
cudaError_t run_ms(const DslashParams &P, const void *Ti, const Spinor &p0, const Spinor &p1, const Spinor &q,
                   const Spinor &tmp, const void *ring, const void *x, const void *dir, int nshift,
                   MultishiftState *state, double *partials, unsigned int *arrived, int *err, BarrierWait wait,
                   int blocks, int steps, const GaugeT &U, cudaStream_t st)
{
    PersistMsArg<GaugeT> a{P.g,
                           U,
                           (const double2 *)P.clover,
                           (const double2 *)Ti,
                           P.b,
                           P.sigma,
                           (const SpinorD *)ring,
                           (const SpinorD *)x,
                           (const SpinorD *)dir,
                           {p0.d(), p1.d()},
                           q.d(),
                           tmp.v ? tmp.d() : SpinorD{},
                           state,
                           partials,
                           arrived,
                           err,
                           wait,
                           nshift,
                           steps};
    const cudaError_t e = cudaMemsetAsync(arrived, 0, sizeof(unsigned int), st);
    if (e != cudaSuccess) return e;
    void *args[] = {&a};
    return cudaLaunchCooperativeKernel((const void *)ms_persist_kernel<EO, GaugeT>, dim3(blocks), dim3(kSplitThreads),
                                       args, 0, st);
}

// The grid of the one-launch multishift: a tile of either parity each, at most as many blocks as are
// resident at once.  0 where these have more than a tile of each parity: a phase then takes two
// rounds (even-odd 12^3 x 24, 648 tiles on 592 blocks: 1.28 times the launches per step).
template <bool EO, class GaugeT> int ms_blocks(const Geom &g, int device)
{
    int sms = 0, coop = 0, per = 0;
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device) != cudaSuccess ||
        cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, device) != cudaSuccess || !coop ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, ms_persist_kernel<EO, GaugeT>, kSplitThreads, 0) !=
            cudaSuccess)
        return 0;
    const int tiles = (g.Vh + kSplitSites - 1) / kSplitSites;
    if (tiles > sms * per) return 0;
    return 2 * tiles < sms * per ? 2 * tiles : sms * per;
}

}  // namespace

int cg_persist_residency(const Geom &g, int rep, int device)
{
    return rep == REP_SU3 ? residency<GaugeD18>(g, device) : residency<GaugeD9>(g, device);
}
int cg_persist_partials(const Geom &g) { return 2 * persist_blocks(g); }

cudaError_t launch_cg_persist(const DslashParams &P, int minb, const Spinor &p0, const Spinor &p1, const Spinor &x,
                              const Spinor &r, const Spinor &q, void *state, double *partials, unsigned int *arrived,
                              int *err, BarrierWait wait, int steps, cudaStream_t st)
{
    const int s = P.g.stride;
    CGState *cs = (CGState *)state;
    if (P.rep == REP_SU3)
        return run(P, minb, p0, p1, x, r, q, cs, partials, arrived, err, wait, steps,
                   GaugeD18{(const double2 *)P.U->d64, s}, st);
    return run(P, minb, p0, p1, x, r, q, cs, partials, arrived, err, wait, steps, GaugeD9{(const double *)P.U->d64, s}, st);
}

int ms_persist_blocks(const Geom &g, int rep, int device, bool even_odd)
{
    if (rep == REP_SU3) return even_odd ? ms_blocks<true, GaugeD18>(g, device) : ms_blocks<false, GaugeD18>(g, device);
    return even_odd ? ms_blocks<true, GaugeD9>(g, device) : ms_blocks<false, GaugeD9>(g, device);
}

cudaError_t launch_ms_persist(const DslashParams &P, const void *Ti, bool even_odd, const Spinor &p0, const Spinor &p1,
                              const Spinor &q, const Spinor &tmp, const void *ring, const void *x, const void *dir,
                              int nshift, void *state, double *partials, unsigned int *arrived, int *err,
                              BarrierWait wait, int blocks, int steps, cudaStream_t st)
{
    const int s = P.g.stride;
    auto go = [&](const auto &U) {
        MultishiftState *ms = (MultishiftState *)state;
        return even_odd ? run_ms<true>(P, Ti, p0, p1, q, tmp, ring, x, dir, nshift, ms, partials, arrived, err, wait,
                                       blocks, steps, U, st)
                        : run_ms<false>(P, Ti, p0, p1, q, tmp, ring, x, dir, nshift, ms, partials, arrived, err, wait,
                                        blocks, steps, U, st);
    };
    return P.rep == REP_SU3 ? go(GaugeD18{(const double2 *)P.U->d64, s}) : go(GaugeD9{(const double *)P.U->d64, s});
}

}  // namespace lym
