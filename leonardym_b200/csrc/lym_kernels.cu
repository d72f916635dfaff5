// Device kernels: layout conversion, gauge upload / compression, clover build,
// and the dispatcher over the stencil instantiations.
#include "lym_blas.cuh"
#include "lym_dslash.cuh"
#include "lym_internal.h"
#include "lym_solver_ops.cuh"

namespace lym {

size_t Spinor::bytes_per_parity() const
{
    switch (prec) {
    case PREC_D: return (size_t)12 * stride * sizeof(double2);
    case PREC_F: return (size_t)6 * stride * sizeof(float4);
    default: return (size_t)3 * stride * sizeof(int4);
    }
}

Spinor Spinor::parity(int p) const
{
    Spinor s = *this;
    s.owned = false;
    s.nparity = 1;
    s.v = (char *)v + (size_t)p * bytes_per_parity();
    if (norm) s.norm = norm + (size_t)p * stride;
    return s;
}

static inline int nblocks(int n, int t) { return (n + t - 1) / t; }

// ----------------------------------------------------------------- layout --
LYM_D void lex_coords(const Geom &g, int s, int c[4])
{
    c[3] = s % g.L[3];
    int r = s / g.L[3];
    c[2] = r % g.L[2];
    r /= g.L[2];
    c[1] = r % g.L[1];
    c[0] = r / g.L[1];
}

template <class View>
__global__ void pack_kernel(Geom g, const double *aos, View v0, View v1)
{
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= g.V) return;
    int c[4];
    lex_coords(g, s, c);
    const int p = (c[0] + c[1] + c[2] + c[3]) & 1;
    cx<double> x[12];
    const double2 *src = reinterpret_cast<const double2 *>(aos) + (size_t)s * 12;
#pragma unroll
    for (int k = 0; k < 12; ++k) {
        double2 w = src[k];
        x[k] = {w.x, w.y};
    }
    (p ? v1 : v0).template store<double>(s >> 1, x);
}

template <class View>
__global__ void unpack_kernel(Geom g, View v0, View v1, double *aos)
{
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= g.V) return;
    int c[4];
    lex_coords(g, s, c);
    const int p = (c[0] + c[1] + c[2] + c[3]) & 1;
    cx<double> x[12];
    (p ? v1 : v0).template load<double>(s >> 1, x);
    double2 *dst = reinterpret_cast<double2 *>(aos) + (size_t)s * 12;
#pragma unroll
    for (int k = 0; k < 12; ++k) dst[k] = make_double2(x[k].re, x[k].im);
}

// FP64: a block takes 16 half-sites of both parities, 32 consecutive sites of the AoS vector, and
// turns them in shared memory, so that reads are 256-byte and writes 6-KB pieces (one thread
// per site writes 16 bytes of a sector at a time: 112 us at 24^3 x 48; 3.8 against 4.9 us at
// 10 x 12 x 14 x 18).
__global__ void __launch_bounds__(128) unpack_tile_kernel(Geom g, SpinorD v0, SpinorD v1, double2 *aos)
{
    constexpr int kWord = 13;  // 12 words of a site, 1 of padding
    __shared__ __align__(16) double2 tile[32 * kWord];
    const int hl = threadIdx.x & 15, p = (threadIdx.x >> 4) & 1, w0 = threadIdx.x >> 5;
    const int h = blockIdx.x * 16 + hl;
    if (h < g.Vh) {
        int c[4];
        site_coords(g, h, p, c);
        double2 *t = tile + (2 * hl + (c[3] & 1)) * kWord;
        const SpinorD &v = p ? v1 : v0;
#pragma unroll
        for (int w = w0; w < 12; w += 4) t[w] = __ldg(v.v + (size_t)w * v.stride + h);
    }
    __syncthreads();
    const int n = min(32, g.V - (int)blockIdx.x * 32) * 12;
    for (int i = threadIdx.x; i < n; i += 128) aos[(size_t)blockIdx.x * 384 + i] = tile[i / 12 * kWord + i % 12];
}

void launch_pack(const Geom &g, const double *aos, const Spinor &full, cudaStream_t st)
{
    const int nb = nblocks(g.V, 128);
    if (full.prec == PREC_D) pack_kernel<<<nb, 128, 0, st>>>(g, aos, full.d(0), full.d(1));
    else if (full.prec == PREC_F) pack_kernel<<<nb, 128, 0, st>>>(g, aos, full.f(0), full.f(1));
    else pack_kernel<<<nb, 128, 0, st>>>(g, aos, full.h(0), full.h(1));
}

void launch_unpack(const Geom &g, const Spinor &full, double *aos, cudaStream_t st)
{
    const int nb = nblocks(g.V, 128);
    if (full.prec == PREC_D) unpack_tile_kernel<<<nblocks(g.V, 32), 128, 0, st>>>(g, full.d(0), full.d(1), (double2 *)aos);
    else if (full.prec == PREC_F) unpack_kernel<<<nb, 128, 0, st>>>(g, full.f(0), full.f(1), aos);
    else unpack_kernel<<<nb, 128, 0, st>>>(g, full.h(0), full.h(1), aos);
}

template <class Dst, class Src>
__global__ void convert_kernel(int vh, Dst d, Src s)
{
    const int h = blockIdx.x * blockDim.x + threadIdx.x;
    if (h >= vh) return;
    cx<double> x[12];
    s.template load<double>(h, x);
    d.template store<double>(h, x);
}

template <class Dst>
static void convert_from(const Geom &g, const Dst &d, const Spinor &src, int p, cudaStream_t st)
{
    const int nb = nblocks(g.Vh, 128);
    if (src.prec == PREC_D) convert_kernel<<<nb, 128, 0, st>>>(g.Vh, d, src.d(p));
    else if (src.prec == PREC_F) convert_kernel<<<nb, 128, 0, st>>>(g.Vh, d, src.f(p));
    else convert_kernel<<<nb, 128, 0, st>>>(g.Vh, d, src.h(p));
}

void launch_convert(const Geom &g, const Spinor &dst, const Spinor &src, cudaStream_t st)
{
    const int np = dst.nparity < src.nparity ? dst.nparity : src.nparity;
    for (int p = 0; p < np; ++p) {
        if (dst.prec == PREC_D) convert_from(g, dst.d(p), src, p, st);
        else if (dst.prec == PREC_F) convert_from(g, dst.f(p), src, p, st);
        else convert_from(g, dst.h(p), src, p, st);
    }
}

// ------------------------------------------------------------------ gauge --
// Fundamental gauge links -> fermion links: the adjoint map for SU(2)
// (utils/ConvertLattice.h:24-34,100-105) and the boundary condition folded into the
// links (LatticeBoundaryConditions.h:8-14).  In/out are host-layout AoS arrays.
__global__ void fundamental_to_fermion_kernel(Geom g, int rep, int bc, const double *gauge, double *fermion)
{
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= g.V) return;
    int c[4];
    lex_coords(g, s, c);
    for (int mu = 0; mu < 4; ++mu) {
        const double sgn = (bc == 1 && mu == 3 && c[3] == g.L[3] - 1) ? -1.0 : 1.0;
        if (rep == REP_SU3) {
            const double *src = gauge + ((size_t)s * 4 + mu) * 18;
            double *dst = fermion + ((size_t)s * 4 + mu) * 18;
            for (int k = 0; k < 18; ++k) dst[k] = sgn * src[k];
        } else {
            // SU(2) column-major complex 2x2 -> real 3x3 adj(a,b) = 2 Re tr(T_a U T_b U^+)
            const double2 *u2 = reinterpret_cast<const double2 *>(gauge) + ((size_t)s * 4 + mu) * 4;
            cx<double> U[2][2] = {{{u2[0].x, u2[0].y}, {u2[2].x, u2[2].y}}, {{u2[1].x, u2[1].y}, {u2[3].x, u2[3].y}}};
            const cx<double> Tm[3][2][2] = {{{{0, 0}, {0.5, 0}}, {{0.5, 0}, {0, 0}}},
                                            {{{0, 0}, {0, -0.5}}, {{0, 0.5}, {0, 0}}},
                                            {{{0.5, 0}, {0, 0}}, {{0, 0}, {-0.5, 0}}}};
            double *dst = fermion + ((size_t)s * 4 + mu) * 9;
            for (int a = 0; a < 3; ++a)
                for (int b = 0; b < 3; ++b) {
                    cx<double> A[2][2], B[2][2];
                    for (int i = 0; i < 2; ++i)
                        for (int j = 0; j < 2; ++j) {
                            A[i][j] = {0, 0};
                            for (int k = 0; k < 2; ++k) fma_c(A[i][j], Tm[a][i][k], U[k][j]);
                        }
                    for (int i = 0; i < 2; ++i)
                        for (int j = 0; j < 2; ++j) {
                            B[i][j] = {0, 0};
                            for (int k = 0; k < 2; ++k) fma_c(B[i][j], A[i][k], Tm[b][k][j]);
                        }
                    double tr = 0.0;
                    for (int i = 0; i < 2; ++i)
                        for (int k = 0; k < 2; ++k) {
                            cx<double> t = B[i][k] * conj(U[i][k]);  // (B U^+)_ii = sum_k B_ik conj(U_ik)
                            tr += t.re;
                        }
                    dst[b * 3 + a] = sgn * 2.0 * tr;
                }
        }
    }
}

void launch_fundamental_to_fermion(const Geom &g, int rep, int bc, const double *gauge_aos, double *fermion_aos,
                                   cudaStream_t st)
{
    fundamental_to_fermion_kernel<<<nblocks(g.V, 128), 128, 0, st>>>(g, rep, bc, gauge_aos, fermion_aos);
}

// --------------------------------------------------------- index checking --
// Reference-order neighbour tables (LocalLayout.h:34-110), for layout tests.
__global__ void neighbour_tables_kernel(Geom g, int *sup, int *sdn)
{
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= g.V) return;
    int c[4];
    lex_coords(g, s, c);
    for (int mu = 0; mu < 4; ++mu) {
        int a[4] = {c[0], c[1], c[2], c[3]}, b[4] = {c[0], c[1], c[2], c[3]};
        a[mu] = (a[mu] + 1) % g.L[mu];
        b[mu] = (b[mu] - 1 + g.L[mu]) % g.L[mu];
        sup[s * 4 + mu] = lex_of(g, a[0], a[1], a[2], a[3]);
        sdn[s * 4 + mu] = lex_of(g, b[0], b[1], b[2], b[3]);
    }
}

void launch_neighbour_tables(const Geom &g, int *sup, int *sdn, cudaStream_t st)
{
    neighbour_tables_kernel<<<nblocks(g.V, 128), 128, 0, st>>>(g, sup, sdn);
}

// What the stencil computes for every (parity, h): its own lexicographic index and
// the half-site indices of its 8 neighbours, out[(p*Vh + h)*9 + k].
__global__ void stencil_index_probe_kernel(Geom g, int *out)
{
    const int h = blockIdx.x * blockDim.x + threadIdx.x;
    const int p = blockIdx.y;
    if (h >= g.Vh) return;
    int c[4];
    site_coords(g, h, p, c);
    int *o = out + ((size_t)p * g.Vh + h) * 9;
    o[0] = lex_of(g, c[0], c[1], c[2], c[3]);
    for (int mu = 0; mu < 4; ++mu) {
        o[1 + 2 * mu] = neighbour_h(g, c, mu, +1);
        o[2 + 2 * mu] = neighbour_h(g, c, mu, -1);
    }
}

__global__ void nbr_table_kernel(Geom g, int *nbr)
{
    const int h = blockIdx.x * blockDim.x + threadIdx.x;
    const int p = blockIdx.y;
    if (h >= g.Vh) return;
    int c[4];
    site_coords(g, h, p, c);
    for (int mu = 0; mu < 4; ++mu) {
        nbr[(size_t)(p * 8 + 2 * mu) * g.stride + h] = neighbour_h(g, c, mu, +1);
        nbr[(size_t)(p * 8 + 2 * mu + 1) * g.stride + h] = neighbour_h(g, c, mu, -1);
    }
}

void launch_nbr_table(const Geom &g, int *nbr, cudaStream_t st)
{
    dim3 grid(nblocks(g.Vh, 128), 2);
    nbr_table_kernel<<<grid, 128, 0, st>>>(g, nbr);
}

void launch_stencil_index_probe(const Geom &g, int *out, cudaStream_t st)
{
    dim3 grid(nblocks(g.Vh, 128), 2);
    stencil_index_probe_kernel<<<grid, 128, 0, st>>>(g, out);
}

// ----------------------------------------------------------------- dslash --
template <typename R, class S, class G, class C>
static void run_dslash(const DslashParams &P, const S &in, const S &out, const S &y, const S &v2, const G &U,
                       const C &T, cudaStream_t st)
{
    DslashArg<S, G, C> a;
    a.g = P.g;
    a.in = in;
    a.out = out;
    a.y = y;
    a.v2 = v2;
    a.U = U;
    a.T = T;
    a.parity = P.parity;
    a.gamma5 = P.gamma5;
    a.has_v2 = P.has_v2;
    a.has_clover = P.clover != nullptr;
    a.a = P.a;
    a.b = P.b;
    a.alpha_re = P.alpha_re;
    a.alpha_im = P.alpha_im;
    a.skip_if = P.skip_if;
    const int nb = nblocks(P.g.Vh, 128);
    switch (P.epi) {
    case EPI_SCALE_: dslash_kernel<R, EPI_SCALE><<<nb, 128, 0, st>>>(a); break;
    case EPI_CLOVINV_: dslash_kernel<R, EPI_CLOVINV><<<nb, 128, 0, st>>>(a); break;
    case EPI_XPAY_: dslash_kernel<R, EPI_XPAY><<<nb, 128, 0, st>>>(a); break;
    default: dslash_kernel<R, EPI_XPAY_INV><<<nb, 128, 0, st>>>(a); break;
    }
}

void launch_dslash(const DslashParams &P, cudaStream_t st)
{
    const GaugeDev &U = *P.U;
    const int s = P.g.stride;
    if (P.prec == PREC_D) {
        launch_split(P, st);
    } else if (P.prec == PREC_F) {
        CloverF T{(const float4 *)P.clover, s};
        if (P.rep == REP_SU3 && U.link_reals == 8)
            run_dslash<float>(P, P.in.f(), P.out.f(), P.y.f(), P.v2.f(), GaugeF8{(const float4 *)U.f32r8, U.sign, s}, T,
                              st);
        else if (P.rep == REP_SU3)
            run_dslash<float>(P, P.in.f(), P.out.f(), P.y.f(), P.v2.f(), GaugeF12{(const float4 *)U.f32, U.sign, s}, T,
                              st);
        else
            run_dslash<float>(P, P.in.f(), P.out.f(), P.y.f(), P.v2.f(), GaugeF6{(const float2 *)U.f32, U.sign, s}, T,
                              st);
    } else {
        CloverH T{(const uint2 *)P.clover, s};
        if (P.rep == REP_SU3)
            run_dslash<float>(P, P.in.h(), P.out.h(), P.y.h(), P.v2.h(), GaugeH12{(const uint2 *)U.h16, U.sign, s}, T,
                              st);
        else
            run_dslash<float>(P, P.in.h(), P.out.h(), P.y.h(), P.v2.h(), GaugeH6{(const __half2 *)U.h16, U.sign, s}, T,
                              st);
    }
}

// ---------------------------------------------------- stencil + CG epilogue --
struct CGAlphaFromNorm {  // alpha = |r|^2 / <p, A p> with <p, A p> = |Q p|^2
    CGState *s;
    LYM_D void operator()(double qq) const { s->alpha = make_double2(s->rr / qq, 0.0); }
};
template <class Upd> struct CGUpdateFin {  // the scalar step of OpCGUpdate
    Upd u;
    LYM_D void operator()(double rr) const
    {
        const double t[1] = {rr};
        u.finalize(t);
    }
};

template <typename R, class S, class SX, class SR, class G, class C>
static void run_dslash_cg(const DslashParams &P, int mode, const S &in, const S &out, const S &y, const S &p,
                          const SX &x, const SR &r, const G &U, const C &T, void *state, double *partials,
                          unsigned int *counter, cudaStream_t st)
{
    DslashArg<S, G, C> a;
    a.g = P.g;
    a.in = in;
    a.out = out;
    a.y = y;
    a.v2 = p;
    a.U = U;
    a.T = T;
    a.parity = P.parity;
    a.gamma5 = 1;
    a.has_v2 = 0;
    a.has_clover = P.clover != nullptr;
    a.a = P.a;
    a.b = P.b;
    a.alpha_re = a.alpha_im = 0.0;
    a.skip_if = P.skip_if;
    CGState *cs = (CGState *)state;
    const int nb = nblocks(P.g.Vh, 128);
    if (mode == CG_NORM) {
        CGEpilogue<SX, SR, CGAlphaFromNorm> f{x, r, &cs->alpha, CGAlphaFromNorm{cs}, partials, counter};
        dslash_cg_kernel<R, CG_NORM><<<nb, 128, 0, st>>>(a, f);
    } else {
        typedef OpCGUpdate<SX, S, SR, S> Upd;
        CGEpilogue<SX, SR, CGUpdateFin<Upd>> f{x, r, &cs->alpha, CGUpdateFin<Upd>{Upd{x, p, r, p, cs}}, partials,
                                                counter};
        dslash_cg_kernel<R, CG_UPDATE><<<nb, 128, 0, st>>>(a, f);
    }
}

void launch_dslash_cg(const DslashParams &P, int mode, const Spinor &p, const Spinor &x, const Spinor &r, void *state,
                      double *partials, unsigned int *counter, cudaStream_t st)
{
    const GaugeDev &U = *P.U;
    const int s = P.g.stride;
    if (P.prec == PREC_D) {
        launch_split_cg(P, mode, p, x, r, state, partials, counter, st);
    } else if (P.prec == PREC_F) {
        CloverF T{(const float4 *)P.clover, s};
        if (P.rep == REP_SU3 && U.link_reals == 8)
            run_dslash_cg<float>(P, mode, P.in.f(), P.out.f(), P.y.f(), p.f(), x.f(), r.f(),
                                 GaugeF8{(const float4 *)U.f32r8, U.sign, s}, T, state, partials, counter, st);
        else if (P.rep == REP_SU3)
            run_dslash_cg<float>(P, mode, P.in.f(), P.out.f(), P.y.f(), p.f(), x.f(), r.f(),
                                 GaugeF12{(const float4 *)U.f32, U.sign, s}, T, state, partials, counter, st);
        else
            run_dslash_cg<float>(P, mode, P.in.f(), P.out.f(), P.y.f(), p.f(), x.f(), r.f(),
                                 GaugeF6{(const float2 *)U.f32, U.sign, s}, T, state, partials, counter, st);
    } else {
        CloverH T{(const uint2 *)P.clover, s};
        if (P.rep == REP_SU3)
            run_dslash_cg<float>(P, mode, P.in.h(), P.out.h(), P.y.h(), p.h(), x.f(), r.f(),
                                 GaugeH12{(const uint2 *)U.h16, U.sign, s}, T, state, partials, counter, st);
        else
            run_dslash_cg<float>(P, mode, P.in.h(), P.out.h(), P.y.h(), p.h(), x.f(), r.f(),
                                 GaugeH6{(const __half2 *)U.h16, U.sign, s}, T, state, partials, counter, st);
    }
}

template <typename R, class S, class C>
static void run_clover(const Geom &g, const S &out, const S &in, const C &T, int parity, int gamma5, cudaStream_t st)
{
    clover_kernel<R><<<nblocks(g.Vh, 128), 128, 0, st>>>(g, out, in, T, parity, gamma5);
}

void launch_clover(const Geom &g, int prec, const Spinor &out, const Spinor &in, const void *clover, int parity,
                   int gamma5, cudaStream_t st)
{
    if (prec == PREC_D) run_clover<double>(g, out.d(), in.d(), CloverD{(const double2 *)clover, g.stride}, parity, gamma5, st);
    else if (prec == PREC_F) run_clover<float>(g, out.f(), in.f(), CloverF{(const float4 *)clover, g.stride}, parity, gamma5, st);
    else run_clover<float>(g, out.h(), in.h(), CloverH{(const uint2 *)clover, g.stride}, parity, gamma5, st);
}

}  // namespace lym
