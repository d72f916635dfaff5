// Launches of the FP64 stencil (lym_split.cuh): operator applications, Schur halves, and the
// products of CG and multishift iterations with their vector work fused.
//
// In "both" mode a launch covers both parities, the same half-sites of either in one block, so
// that a link read forward by one parity and backward by the other comes from DRAM once; it can
// write the result straight into the caller's AoS vector (through shared memory, whole sites).
#include "lym_blas.cuh"
#include "lym_dslash.cuh"
#include "lym_internal.h"
#include "lym_solver_ops.cuh"
#include "lym_split.cuh"

namespace lym {

namespace {

using namespace split;

enum SplitEpi : int {
    SPLIT_SCALE = EPI_SCALE,
    SPLIT_CLOVINV = EPI_CLOVINV,
    SPLIT_XPAY = EPI_XPAY,
    SPLIT_XPAY_INV = EPI_XPAY_INV,
    // CG on A = Q Q + sigma, Q = gamma5 D or gamma5 S (Hermitian): the vector work of an iteration
    // inside its two products, as CG_NORM / CG_UPDATE of lym_dslash.cuh
    SPLIT_CG_NORM = 10,    // q = Q p stored, <p, A p> = |q|^2 + sigma |p|^2 reduced
    SPLIT_CG_UPDATE = 11,  // A p = Q q + sigma p in registers; x += alpha p, r -= alpha A p, |r|^2
    // the second product of a multishift step: r_{k+1} = r_k - alpha A p in a ring of residuals
    SPLIT_MS_RESIDUAL = 12,
};

template <class GaugeT> struct SplitArg {
    Geom g;
    SpinorD in[2], out[2], y[2], v2[2], x[2], r[2];  // by output parity
    GaugeT U;
    const double2 *clover;
    int parity;  // 0, 1, or 2: both
    int gamma5, has_v2;
    double a, b, alpha_re, alpha_im;
    const int *skip_if;
    int *on_skip;            // SPLIT_CG_NORM: set when the launch is skipped
    const double2 *aos_in;   // IN_AOS
    double2 *aos_out;        // AOS: the full result
    const double2 *aos_v2;   // AOS: the added vector, or null
    int even_identity;       // both mode: no stencil on the even sites (AOS: they get y; in
                             // the CG modes A is 1 + sigma there)
    double sigma;            // SPLIT_CG_*
    const double2 *alpha;    // SPLIT_CG_UPDATE
    const SpinorD *ring;     // SPLIT_MS_RESIDUAL: kMsWin + 1 full spinors
    const MultishiftState *ms;
    double *partials;        // SPLIT_CG_*: [gridDim.x]
    unsigned int *counter;
};

struct NoFin {
    LYM_D void operator()(double) const {}
};
struct AlphaFin {  // alpha = |r|^2 / <p, A p>
    CGState *s;
    LYM_D void operator()(double pap) const { s->alpha = make_double2(s->rr / pap, 0.0); }
};
struct MsAlphaFin {
    static constexpr bool kParallelFinalize = true;
    MultishiftState *s;
    LYM_D void operator()(double pap) const { ms_alpha_step(s, pap); }
};
struct MsResidualFin {
    MultishiftState *s;
    static constexpr bool kParallelFinalize = true;
    LYM_D void operator()(double rr) const { ms_residual_step(s, rr); }
};
struct UpdateFin {  // the scalar step of OpCGUpdate
    CGState *s;
    LYM_D void operator()(double rr) const
    {
        const double t[1] = {rr};
        OpCGUpdate<SpinorD, SpinorD, SpinorD, SpinorD> u{SpinorD{}, SpinorD{}, SpinorD{}, SpinorD{}, s};
        u.finalize(t);
    }
};

// where a launch reads its input: packed spinors, or (SPLIT_XPAY to AoS) the caller's AoS vector
enum SplitIn : int { IN_PACKED = 0, IN_AOS = 1 };
LYM_D C load_aos(const double2 *v, int word, int s)
{
    const double2 w = __ldg(v + (size_t)s * 12 + word);
    return C{w.x, w.y};
}

// a word of a vector that the same launch writes (load1 reads through the path for data that nothing
// writes meanwhile)
LYM_D C load_own(const SpinorD &v, int word, int h)
{
    const double2 w = v.v[(size_t)word * v.stride + h];
    return C{w.x, w.y};
}

template <int EPI, bool AOS, int IN, class GaugeT, class Fin>
__global__ void __launch_bounds__(kSplitThreads, 4) split_kernel(const SplitArg<GaugeT> arg, const Fin fin)
{
    if (arg.skip_if && *arg.skip_if) {
        if (EPI == SPLIT_CG_NORM && arg.on_skip && blockIdx.x == 0 && threadIdx.x == 0) *arg.on_skip = 1;
        return;
    }
    constexpr bool kSecond = EPI == SPLIT_CG_UPDATE || EPI == SPLIT_MS_RESIDUAL;  // A p stays in registers
    constexpr bool kReduce = EPI == SPLIT_CG_NORM || kSecond;
    constexpr bool kXpay = EPI == SPLIT_XPAY || kReduce;
    constexpr int kTileWord = 13;  // 12 words of a site, 1 of padding
    __shared__ __align__(16) double2 tile[AOS ? kSplitSites * kTileWord : 1];
    const Geom &g = arg.g;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int d = (lane >> 3) & 1, k = lane >> 4;
    int p, hr;
    if (kReduce && arg.even_identity) {
        // the stencil's blocks, 32 odd half-sites each, then those of the even sites, which only
        // stream: with both parities in a block half of its warps would idle (10 x 12 x 14 x 18,
        // multishift: 1.0 us of the norm's launch and 2.0 us of the residual's; these take 15.1 and
        // 16.7 us at 12^3 x 24)
        const int odd = (g.Vh + kSplitSites - 1) / kSplitSites, blk = blockIdx.x;
        p = blk < odd ? 1 : 0;
        hr = (p ? blk : blk - odd) * kSplitSites + warp * 8 + (lane & 7);
    } else if (arg.parity == 2) {
        p = warp >> 1;
        hr = blockIdx.x * (kSplitSites / 2) + (warp & 1) * 8 + (lane & 7);
    } else {
        p = arg.parity;
        hr = blockIdx.x * kSplitSites + warp * 8 + (lane & 7);
    }
    const bool in = hr < g.Vh;
    const int h = in ? hr : g.Vh - 1;
    if (AOS && arg.aos_v2) {
        for (int i = threadIdx.x; i < kSplitSites * 12; i += kSplitThreads) {
            const int site = i / 12;
            if (blockIdx.x * kSplitSites + site < g.V)
                copy16(tile + site * kTileWord + i % 12, arg.aos_v2 + (size_t)blockIdx.x * kSplitSites * 12 + i);
        }
    }
    int c[4];
    site_coords(g, h, p, c);
    const int s = lex_of(g, c[0], c[1], c[2], c[3]);
    const int sp = 3 * (2 * d + k), so = 3 * (2 * d + 1 - k);  // words of the own and the other spin
    C res[3];
    C yo[3];  // y (NORM: p) of the own spin
    const bool identity = (AOS || kReduce) && arg.even_identity && p == 0;
    if (identity) {
        if (!kSecond) {
#pragma unroll
            for (int m = 0; m < 3; ++m) res[m] = yo[m] = load1(arg.y[0], sp + m, h);
        }
    } else {
        const double2 *const clover = arg.clover + (size_t)((p * 2 + d) * 18) * g.stride + h;
        auto word = [&](int w) { return __ldg(clover + (size_t)clover_word(w, k) * g.stride); };
        C acc[3];
        if constexpr (IN == IN_AOS) {
            split_hopping(g, [&](int w, int sn) { return load_aos(arg.aos_in, w, sn); }, arg.U, p, h, s, c, k, d, acc);
        } else {
            const SpinorD x = arg.in[p];
            split_hopping(g, [&](int w, int sn) { return load1(x, w, sn >> 1); }, arg.U, p, h, s, c, k, d, acc);
        }
        // y of the site: an AoS input is its own y
        auto y = [&](int w) { return IN == IN_AOS ? load_aos(arg.aos_in, w, s) : load1(arg.y[p], w, h); };
        C own[3], oth[3];
        if constexpr (EPI == SPLIT_SCALE) {
#pragma unroll
            for (int m = 0; m < 3; ++m) res[m] = arg.a * acc[m];
        } else if constexpr (EPI == SPLIT_CLOVINV || EPI == SPLIT_XPAY_INV) {
#pragma unroll
            for (int m = 0; m < 3; ++m) {
                if (EPI == SPLIT_CLOVINV) {
                    own[m] = arg.a * acc[m];
                } else {
                    own[m] = y(sp + m);
                    fma_r(own[m], arg.b, acc[m]);
                }
                oth[m] = shfl_xor(own[m], 16);
            }
            clover_rows(word, k, own, oth, res);
        } else {
#pragma unroll
            for (int m = 0; m < 3; ++m) yo[m] = own[m] = y(sp + m);
            if (arg.clover) {
#pragma unroll
                for (int m = 0; m < 3; ++m) oth[m] = y(so + m);
                clover_rows(word, k, own, oth, res);
            } else {
#pragma unroll
                for (int m = 0; m < 3; ++m) res[m] = own[m];
            }
#pragma unroll
            for (int m = 0; m < 3; ++m) {
                fma_r(res[m], arg.b, acc[m]);
                if (d && arg.gamma5) res[m] = -res[m];
            }
        }
    }
    if constexpr (kXpay && !kReduce && !AOS) {
        if (arg.has_v2) {
            const C al = {arg.alpha_re, arg.alpha_im};
#pragma unroll
            for (int m = 0; m < 3; ++m) fma_c(res[m], al, load1(arg.v2[p], sp + m, h));
        }
    }
    if constexpr (AOS) {
        double2 *t = tile + (s - blockIdx.x * kSplitSites) * kTileWord + sp;
        if (arg.aos_v2) {
            asm volatile("cp.async.wait_all;\n" ::: "memory");
            __syncthreads();
            const C al = {arg.alpha_re, arg.alpha_im};
            if (in) {
#pragma unroll
                for (int m = 0; m < 3; ++m) fma_c(res[m], al, C{t[m].x, t[m].y});
            }
        }
        if (in) {
#pragma unroll
            for (int m = 0; m < 3; ++m) t[m] = make_double2(res[m].re, res[m].im);
        }
        __syncthreads();
        for (int i = threadIdx.x; i < kSplitSites * 12; i += kSplitThreads) {
            const int site = i / 12;
            if (blockIdx.x * kSplitSites + site < g.V)
                arg.aos_out[(size_t)blockIdx.x * kSplitSites * 12 + i] = tile[site * kTileWord + i % 12];
        }
        return;
    }
    double part = 0.0;
    if (in) {
        auto put = [&](const SpinorD &v, int m, C z) {
            v.v[(size_t)(sp + m) * v.stride + h] = make_double2(z.re, z.im);
        };
        if constexpr (EPI == SPLIT_CG_UPDATE) {
            const double2 al2 = *arg.alpha;
            const C al = {al2.x, al2.y};
            C pv[3], xv[3], rv[3];  // all read before the first is written
#pragma unroll
            for (int m = 0; m < 3; ++m) {
                pv[m] = load1(arg.v2[p], sp + m, h);
                xv[m] = load_own(arg.x[p], sp + m, h);
                rv[m] = load_own(arg.r[p], sp + m, h);
            }
#pragma unroll
            for (int m = 0; m < 3; ++m) {
                C ap = identity ? pv[m] : res[m];
                fma_c(xv[m], al, pv[m]);
                fma_r(ap, arg.sigma, pv[m]);
                rv[m] = rv[m] - al * ap;
                part += rv[m].re * rv[m].re + rv[m].im * rv[m].im;
                put(arg.x[p], m, xv[m]);
                put(arg.r[p], m, rv[m]);
            }
        } else if constexpr (EPI == SPLIT_MS_RESIDUAL) {
            const int it = arg.ms->iter;
            const SpinorD rin = arg.ring[it % (kMsWin + 1)].par(p), rout = arg.ring[(it + 1) % (kMsWin + 1)].par(p);
            const double al = arg.ms->alpha;
            C pv[3], rv[3];  // rin may be rout
#pragma unroll
            for (int m = 0; m < 3; ++m) {
                pv[m] = load1(arg.v2[p], sp + m, h);
                rv[m] = load_own(rin, sp + m, h);
            }
#pragma unroll
            for (int m = 0; m < 3; ++m) {
                C ap = identity ? pv[m] : res[m];
                fma_r(ap, arg.sigma, pv[m]);
                fma_r(rv[m], -al, ap);
                part += rv[m].re * rv[m].re + rv[m].im * rv[m].im;
                put(rout, m, rv[m]);
            }
        } else {
            double pp = 0.0;
#pragma unroll
            for (int m = 0; m < 3; ++m) {
                if (!identity) put(arg.out[p], m, res[m]);
                if (kReduce) {
                    part += res[m].re * res[m].re + res[m].im * res[m].im;
                    pp += yo[m].re * yo[m].re + yo[m].im * yo[m].im;
                }
            }
            if (kReduce && arg.sigma != 0.0) part += arg.sigma * pp;
        }
    }
    if constexpr (kReduce) {
        // fixed-order reduction: warps, the block's warps, then the blocks in order
        __shared__ double wsum[kSplitThreads / 32];
        __shared__ bool last;
        auto block_total = [&](double v) {
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
            if (lane == 0) wsum[warp] = v;
            __syncthreads();
            return (wsum[0] + wsum[1]) + (wsum[2] + wsum[3]);
        };
        const double tot = block_total(part);
        if (threadIdx.x == 0) {
            arg.partials[blockIdx.x] = tot;
            __threadfence();
            last = atomicAdd(arg.counter, 1u) == gridDim.x - 1;
        }
        __syncthreads();
        if (!last) return;
        __threadfence();
        double t = 0.0;
#pragma unroll 8
        for (int i = threadIdx.x; i < (int)gridDim.x; i += kSplitThreads) t += __ldcg(arg.partials + i);
        const double all = block_total(t);
        if (ParallelFinalize<Fin>::value || threadIdx.x == 0) fin(all);
        if (threadIdx.x == 0) *arg.counter = 0u;
    }
}

template <class GaugeT> SplitArg<GaugeT> split_arg(const DslashParams &P, const GaugeT &U)
{
    SplitArg<GaugeT> a;
    a.g = P.g;
    a.U = U;
    a.parity = P.parity;
    // views of one parity, or of the full spinors in both mode
    const bool both = P.parity == 2 && !P.even_identity;
    for (int p = 0; p < 2; ++p) {
        a.in[p] = P.in.v ? (both ? P.in.d(1 - p) : P.in.d()) : SpinorD{};
        a.out[p] = P.out.v ? (both ? P.out.d(p) : P.out.d()) : SpinorD{};
        a.y[p] = P.y.v ? (both ? P.y.d(p) : P.y.d()) : SpinorD{};
        a.v2[p] = P.v2.v ? (both ? P.v2.d(p) : P.v2.d()) : SpinorD{};
        a.x[p] = a.r[p] = SpinorD{};
    }
    if (P.even_identity) a.y[0] = P.even.d();
    a.clover = (const double2 *)P.clover;
    a.gamma5 = P.gamma5;
    a.has_v2 = P.has_v2;
    a.a = P.a;
    a.b = P.b;
    a.alpha_re = P.alpha_re;
    a.alpha_im = P.alpha_im;
    a.skip_if = P.skip_if;
    a.on_skip = nullptr;
    a.aos_in = (const double2 *)P.aos_in;
    a.aos_out = (double2 *)P.aos_out;
    a.aos_v2 = (const double2 *)P.aos_v2;
    a.even_identity = P.even_identity;
    a.sigma = P.sigma;
    a.alpha = nullptr;
    a.ring = nullptr;
    a.ms = nullptr;
    a.partials = nullptr;
    a.counter = nullptr;
    return a;
}

// even_identity with sums: odd and even half-sites in blocks of their own
int split_blocks(const Geom &g, int parity, bool apart = false)
{
    if (apart) return 2 * ((g.Vh + kSplitSites - 1) / kSplitSites);
    const int per = parity == 2 ? kSplitSites / 2 : kSplitSites;
    return (g.Vh + per - 1) / per;
}

template <class GaugeT> void run_split(const DslashParams &P, const GaugeT &U, cudaStream_t st)
{
    const SplitArg<GaugeT> a = split_arg(P, U);
    const int nb = split_blocks(P.g, P.parity), nt = kSplitThreads;
    if (P.aos_out) {
        if (P.aos_in) split_kernel<SPLIT_XPAY, true, IN_AOS><<<nb, nt, 0, st>>>(a, NoFin{});
        else split_kernel<SPLIT_XPAY, true, IN_PACKED><<<nb, nt, 0, st>>>(a, NoFin{});
        return;
    }
    switch (P.epi) {
    case EPI_SCALE_: split_kernel<SPLIT_SCALE, false, IN_PACKED><<<nb, nt, 0, st>>>(a, NoFin{}); break;
    case EPI_CLOVINV_: split_kernel<SPLIT_CLOVINV, false, IN_PACKED><<<nb, nt, 0, st>>>(a, NoFin{}); break;
    case EPI_XPAY_: split_kernel<SPLIT_XPAY, false, IN_PACKED><<<nb, nt, 0, st>>>(a, NoFin{}); break;
    default: split_kernel<SPLIT_XPAY_INV, false, IN_PACKED><<<nb, nt, 0, st>>>(a, NoFin{}); break;
    }
}

template <class GaugeT>
void run_split_cg(const DslashParams &P, int mode, const Spinor &p, const Spinor &x, const Spinor &r, CGState *cs,
                  double *partials, unsigned int *counter, const GaugeT &U, cudaStream_t st)
{
    SplitArg<GaugeT> a = split_arg(P, U);
    for (int q = 0; q < 2; ++q) {
        const int v = P.parity == 2 ? q : 0;
        a.v2[q] = p.d(v);
        a.x[q] = x.d(v);
        a.r[q] = r.d(v);
    }
    a.gamma5 = 1;
    a.alpha = &cs->alpha;
    a.partials = partials;
    a.counter = counter;
    const int nb = split_blocks(P.g, P.parity, P.even_identity != 0), nt = kSplitThreads;
    if (mode == CG_NORM) split_kernel<SPLIT_CG_NORM, false, IN_PACKED><<<nb, nt, 0, st>>>(a, AlphaFin{cs});
    else split_kernel<SPLIT_CG_UPDATE, false, IN_PACKED><<<nb, nt, 0, st>>>(a, UpdateFin{cs});
}

template <class GaugeT>
void run_split_ms(const DslashParams &P, int mode, const Spinor &p, const SpinorD *ring, MultishiftState *ms,
                  double *partials, unsigned int *counter, const GaugeT &U, cudaStream_t st)
{
    SplitArg<GaugeT> a = split_arg(P, U);
    for (int q = 0; q < 2; ++q) a.v2[q] = p.d(q);
    a.gamma5 = 1;
    a.ring = ring;
    a.ms = ms;
    a.on_skip = &ms->pause;
    a.partials = partials;
    a.counter = counter;
    const int nb = split_blocks(P.g, P.parity, P.even_identity != 0), nt = kSplitThreads;
    if (mode == CG_NORM) split_kernel<SPLIT_CG_NORM, false, IN_PACKED><<<nb, nt, 0, st>>>(a, MsAlphaFin{ms});
    else split_kernel<SPLIT_MS_RESIDUAL, false, IN_PACKED><<<nb, nt, 0, st>>>(a, MsResidualFin{ms});
}

}  // namespace

int split_partials(const Geom &g) { return split_blocks(g, 2, true); }

void launch_split(const DslashParams &P, cudaStream_t st)
{
    const int s = P.g.stride;
    if (P.rep == REP_SU3) run_split(P, GaugeD18{(const double2 *)P.U->d64, s}, st);
    else run_split(P, GaugeD9{(const double *)P.U->d64, s}, st);
}

void launch_split_cg(const DslashParams &P, int mode, const Spinor &p, const Spinor &x, const Spinor &r, void *state,
                     double *partials, unsigned int *counter, cudaStream_t st)
{
    const int s = P.g.stride;
    if (P.rep == REP_SU3)
        run_split_cg(P, mode, p, x, r, (CGState *)state, partials, counter, GaugeD18{(const double2 *)P.U->d64, s}, st);
    else
        run_split_cg(P, mode, p, x, r, (CGState *)state, partials, counter, GaugeD9{(const double *)P.U->d64, s}, st);
}

void launch_split_ms(const DslashParams &P, int mode, const Spinor &p, const void *ring, void *state, double *partials,
                     unsigned int *counter, cudaStream_t st)
{
    const int s = P.g.stride;
    const SpinorD *rv = (const SpinorD *)ring;
    MultishiftState *ms = (MultishiftState *)state;
    if (P.rep == REP_SU3)
        run_split_ms(P, mode, p, rv, ms, partials, counter, GaugeD18{(const double2 *)P.U->d64, s}, st);
    else
        run_split_ms(P, mode, p, rv, ms, partials, counter, GaugeD9{(const double *)P.U->d64, s}, st);
}

}  // namespace lym
