// New gauge fields on the device: the resident link formats of an uploaded field, and the clover
// term T with its even-even inverse, each in one launch.
#include "lym_internal.h"
#include "lym_mat3.cuh"

namespace lym {

namespace {

constexpr int kSites = 32;  // sites of a block of either kernel

LYM_D uint2 halves(double2 a, double2 b)
{
    uint2 w;
    __half2 *hp = reinterpret_cast<__half2 *>(&w);
    hp[0] = __floats2half2_rn((float)a.x, (float)a.y);
    hp[1] = __floats2half2_rn((float)b.x, (float)b.y);
    return w;
}
LYM_D float4 floats(double2 a, double2 b) { return make_float4(a.x, a.y, b.x, b.y); }

// ------------------------------------------------------------------ links --
// AoS input: per site 4 links, each 3 x 3 column-major (complex or real).  A block copies 32
// consecutive sites, contiguous in the input, to shared memory; warp mu then takes link mu of
// each site and writes every resident format: FP64, FP32 in 12 (6) reals, FP16, and for SU(3)
// FP32 in 18 reals.  A link is accepted for the reconstructed formats when it is +-V with V
// special unitary (SU(3)) or special orthogonal (adjoint); the sign goes to the sign table.
// Bound by HBM: 576 bytes a site read and 1184 written (SU(3)).
template <class T> __global__ void __launch_bounds__(128) store_gauge_kernel(Geom g, const T *aos, GaugeDev U, int *err)
{
    constexpr bool kComplex = sizeof(T) == 16;
    constexpr int kSite = 36 + 1;  // elements of a site, padded: conflict-free reads
    __shared__ T sm[kSites * kSite];
    __shared__ unsigned bits[kSites];
    const int s0 = blockIdx.x * kSites, n = min(kSites, g.V - s0);
    if (threadIdx.x < kSites) bits[threadIdx.x] = 0u;
    for (int k = threadIdx.x; k < n * 36; k += 128) sm[k / 36 * kSite + k % 36] = __ldg(aos + (size_t)s0 * 36 + k);
    __syncthreads();
    const int lane = threadIdx.x & 31, mu = threadIdx.x >> 5, s = s0 + lane;
    int c[4];
    coords_of(g, min(s, g.V - 1), c);
    const int p = (c[0] + c[1] + c[2] + c[3]) & 1, h = s >> 1;
    const size_t st = g.stride;
    if (s < g.V) {
        const T *src = sm + lane * kSite + mu * 9;
        Mat<Cd> M;
#pragma unroll
        for (int k = 0; k < 9; ++k) {
            const T v = src[(k % 3) * 3 + k / 3];  // U(i, j) at j * 3 + i
            reinterpret_cast<T *>(U.d64)[((size_t)(p * 4 + mu) * 9 + k) * st + h] = v;
            if constexpr (kComplex) M.a[k / 3][k % 3] = Cd{v.x, v.y};
            else M.a[k / 3][k % 3] = Cd{v, 0.0};
        }
        // unitarity: max |U U^+ - 1|
        double dev = 0.0;
#pragma unroll
        for (int i = 0; i < 3; ++i)
#pragma unroll
            for (int j = 0; j < 3; ++j) {
                Cd a = {i == j ? -1.0 : 0.0, 0.0};
#pragma unroll
                for (int k = 0; k < 3; ++k) fma_c(a, M.a[i][k], conj(M.a[j][k]));
                dev = fmax(dev, fabs(a.re) + fabs(a.im));
            }
        const Cd det = M.a[0][0] * (M.a[1][1] * M.a[2][2] - M.a[1][2] * M.a[2][1]) -
                       M.a[0][1] * (M.a[1][0] * M.a[2][2] - M.a[1][2] * M.a[2][0]) +
                       M.a[0][2] * (M.a[1][0] * M.a[2][1] - M.a[1][1] * M.a[2][0]);
        int neg = 0;
        if (fabs(det.re - 1.0) + fabs(det.im) < 1e-8) neg = 0;
        else if (fabs(det.re + 1.0) + fabs(det.im) < 1e-8) neg = 1;
        else atomicOr(err, 1);
        if (dev > 1e-8) atomicOr(err, 2);
        if (neg) atomicOr(&bits[lane], 1u << mu);
        const size_t w0 = (size_t)(p * 4 + mu) * 3 * st + h;
        auto el = [&](int k) { return make_double2(M.a[k / 3][k % 3].re, M.a[k / 3][k % 3].im); };
        if constexpr (kComplex) {
            float4 *F = reinterpret_cast<float4 *>(U.f32);
            uint2 *H = reinterpret_cast<uint2 *>(U.h16);
            float4 *F18 = reinterpret_cast<float4 *>(U.f32r18) + (size_t)(p * 4 + mu) * 5 * st + h;
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                F[w0 + k * st] = floats(el(2 * k), el(2 * k + 1));
                H[w0 + k * st] = halves(el(2 * k), el(2 * k + 1));
            }
            // all 18 reals (GaugeF18P): entries row-major, two per word, the last word half used
#pragma unroll
            for (int k = 0; k < 5; ++k) F18[k * st] = floats(el(2 * k), k < 4 ? el(2 * k + 1) : make_double2(0.0, 0.0));
        } else {
            float2 *F = reinterpret_cast<float2 *>(U.f32);
            __half2 *H = reinterpret_cast<__half2 *>(U.h16);
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                const float a = (float)el(2 * k).x, b = (float)el(2 * k + 1).x;
                F[w0 + k * st] = make_float2(a, b);
                H[w0 + k * st] = __floats2half2_rn(a, b);
            }
        }
    }
    __syncthreads();
    if (mu == 0 && s < g.V) U.sign[(size_t)p * st + h] = (uint8_t)bits[lane];
}

// 8 reals of V = s U (GaugeF8): (a2, a3), (b1, arg a1, arg c1)
__global__ void __launch_bounds__(128) store_gauge8_kernel(Geom g, GaugeDev U)
{
    const int h = blockIdx.x * blockDim.x + threadIdx.x, p = blockIdx.y, mu = blockIdx.z;
    if (h >= g.Vh) return;
    const Mat<Cd> M = load_link(GaugeD18{(const double2 *)U.d64, g.stride}, p, mu, h);
    const double sg = (U.sign[(size_t)p * g.stride + h] >> mu) & 1 ? -1.0 : 1.0;
    float4 *w = reinterpret_cast<float4 *>(U.f32r8) + (size_t)(p * 4 + mu) * 2 * g.stride + h;
    w[0] = make_float4(sg * M.a[0][1].re, sg * M.a[0][1].im, sg * M.a[0][2].re, sg * M.a[0][2].im);
    w[g.stride] = make_float4(sg * M.a[1][0].re, sg * M.a[1][0].im, atan2(sg * M.a[0][0].im, sg * M.a[0][0].re),
                              atan2(sg * M.a[2][0].im, sg * M.a[2][0].re));
}

// ----------------------------------------------------------------- clover --
// Field strength F_{mu nu} (ImprovedDiracWilsonOperator.cpp:502-523) and the two Hermitian
// blocks of T = 1 + kappa csw gamma5 C with their inverses
// (EvenOddImprovedDiracWilsonOperator.cpp:285-317), in FP64, FP32 and FP16.
//
// clover_build_kernel: one block takes 32 half-sites of one parity.
//   1. Warp pl forms plane pl of each site.  The leaves pair up under F = (Q - Q^+) / 8: a leaf
//      that ends in U_mu(x)^+ contributes minus the leaf that starts with U_mu(x) would, so the
//      two leaves at U_mu(x) are one product U_mu(x) (A - B) of staples, and those at U_mu(x-mu)
//      another: 10 matrix products a plane instead of 12.  F is anti-Hermitian: 9 reals.
//   2. The entries of T from the six planes, in shared memory.
//   3. All words of T in the three precisions, coalesced.
// Bound by the latency of FP64 arithmetic and of the links' loads in 1: 12 warps per SM (168
// registers), FP64 pipe 28 %, DRAM 19 %, 4.3 of 9.3 stall cycles on loads at 20^3 x 40.
// clover_invert_kernel: a thread inverts one block by symmetric sweeps of its packed triangle,
// in registers.  They need no pivoting while the block is positive definite (it is 1 plus the
// clover term, so it is but for a very large kappa c_sw); a block with a pivot that is not
// positive is inverted by Gauss-Jordan with partial pivoting in local memory.  HBM bound.
// A launch of its own because its dependent steps want many warps, the products many registers:
// in one launch they took 532 us at 20^3 x 40, against 439 + 77 us; one thread per site with all
// matrices in local memory, and a separate pass for the FP32 and FP16 words, 1.77 + 0.10 ms.
struct CloverArg {
    Geom g;
    double kc;
    double2 *T, *Ti;
    float4 *Tf, *Tif;
    uint2 *Th, *Tih;
    double *F;  // optional: the field strength, reference layout
    int *err;
};

constexpr int kCloverThreads = 192, kPad = kSites + 1;

// F_pl(i, j) of a site from its 9 reals: imaginary diagonal, entries (1,0), (2,0), (2,1)
LYM_D Cd plane_entry(const double (*f)[9][kPad], int pl, int i, int j, int lane)
{
    if (i == j) return Cd{0.0, f[pl][i][lane]};
    const int e = i + j - 1;  // (1,0) 0, (2,0) 1, (2,1) 2
    const Cd z{f[pl][3 + 2 * e][lane], f[pl][4 + 2 * e][lane]};
    return i > j ? z : Cd{-z.re, z.im};
}

template <class Gauge> LYM_D void plane_of(const Geom &g, const Gauge &U, const int c[4], int mu, int nu, double f[9])
{
    int q[4], o[4];
    auto at = [&](const int d[4], int dir) {
        const Site s = site_of(g, d);
        return load_link(U, s.p, dir, s.h);
    };
    typedef decltype(at(c, 0)) M;
    M R;
    {
        const M Un = at(c, nu);
        moved(g, c, mu, +1, q);
        moved(g, c, nu, +1, o);
        M W = mul(mul(at(q, nu), dag(at(o, mu))), dag(Un));
        moved(g, c, nu, -1, o);
        moved(g, q, nu, -1, q);
        const M B = mul(mul(dag(at(q, nu)), dag(at(o, mu))), at(o, nu));
#pragma unroll
        for (int i = 0; i < 3; ++i)
#pragma unroll
            for (int j = 0; j < 3; ++j) W.a[i][j] = W.a[i][j] - B.a[i][j];
        R = mul(at(c, mu), W);
    }
    {
        const M Un = at(c, nu);
        moved(g, c, mu, -1, q);
        moved(g, q, nu, +1, o);
        M W = mul(mul(Un, dag(at(o, mu))), dag(at(q, nu)));
        moved(g, q, nu, -1, o);
        const M E = mul(dag(at(o, mu)), at(o, nu));
        moved(g, c, nu, -1, o);
        const M B = mul(dag(at(o, nu)), E);
#pragma unroll
        for (int i = 0; i < 3; ++i)
#pragma unroll
            for (int j = 0; j < 3; ++j) W.a[i][j] = W.a[i][j] - B.a[i][j];
        mul_add(R, W, at(q, mu));
    }
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        if constexpr (sizeof(R.a[0][0]) == 16) f[i] = 0.25 * R.a[i][i].im;
        else f[i] = 0.0;
    }
#pragma unroll
    for (int e = 0; e < 3; ++e) {
        const int i = e == 0 ? 1 : 2, j = e == 2 ? 1 : 0;
        const auto z = R.a[i][j] - conj(R.a[j][i]);
        if constexpr (sizeof(z) == 16) {
            f[3 + 2 * e] = 0.125 * z.re;
            f[4 + 2 * e] = 0.125 * z.im;
        } else {
            f[3 + 2 * e] = 0.125 * z;
            f[4 + 2 * e] = 0.0;
        }
    }
}

// The inverse of the packed Hermitian block by Gauss-Jordan with partial pivoting, its Hermitian
// part.  False for a zero pivot.
__device__ __noinline__ bool invert_pivoted(double2 w[18])
{
    Cd m[6][6], inv[6][6];
    for (int i = 0; i < 6; ++i)
        for (int j = 0; j < 6; ++j) {
            inv[i][j] = Cd{i == j ? 1.0 : 0.0, 0.0};
            if (i == j) {
                m[i][j] = Cd{(i & 1) ? w[i >> 1].y : w[i >> 1].x, 0.0};
            } else {
                const double2 z = w[3 + (i > j ? tri_index(i, j) : tri_index(j, i))];
                m[i][j] = Cd{z.x, i > j ? z.y : -z.y};
            }
        }
    for (int col = 0; col < 6; ++col) {
        int piv = col;
        double best = fabs(m[col][col].re) + fabs(m[col][col].im);
        for (int r = col + 1; r < 6; ++r) {
            const double a = fabs(m[r][col].re) + fabs(m[r][col].im);
            if (a > best) {
                best = a;
                piv = r;
            }
        }
        if (best == 0.0) return false;
        const Cd d = m[piv][col];
        const double dn = d.re * d.re + d.im * d.im;
        const Cd rd{d.re / dn, -d.im / dn};
        for (int j = 0; j < 6; ++j) {
            const Cd a = m[piv][j], b = inv[piv][j];
            m[piv][j] = m[col][j];
            inv[piv][j] = inv[col][j];
            m[col][j] = a * rd;
            inv[col][j] = b * rd;
        }
        for (int r = 0; r < 6; ++r) {
            if (r == col) continue;
            const Cd f = m[r][col];
            for (int j = 0; j < 6; ++j) {
                m[r][j] = m[r][j] - f * m[col][j];
                inv[r][j] = inv[r][j] - f * inv[col][j];
            }
        }
    }
    for (int k = 0; k < 3; ++k) w[k] = make_double2(inv[2 * k][2 * k].re, inv[2 * k + 1][2 * k + 1].re);
    for (int i = 1; i < 6; ++i)
        for (int j = 0; j < i; ++j) {
            const Cd z = 0.5 * (inv[i][j] + conj(inv[j][i]));
            w[3 + tri_index(i, j)] = make_double2(z.re, z.im);
        }
    return true;
}

// The inverse of the packed Hermitian block by sweeps: with D = a_kk, a_ij -= a_ik conj(a_jk) / D,
// a_ik /= D, a_kk = -1 / D for k = 0..5 leaves minus the inverse.  False once a pivot is not
// positive (d, l then hold no inverse).
LYM_D bool invert_sweep(double d[6], Cd l[15])
{
    bool ok = true;
#pragma unroll
    for (int k = 0; k < 6; ++k) {
        ok = ok && d[k] > 0.0;
        const double r = 1.0 / d[k];
        Cd b[6], q[6];  // column k, and divided by the pivot
#pragma unroll
        for (int i = 0; i < 6; ++i) {
            if (i == k) continue;
            b[i] = i > k ? l[tri_index(i, k)] : conj(l[tri_index(k, i)]);
            q[i] = r * b[i];
        }
#pragma unroll
        for (int i = 0; i < 6; ++i) {
            if (i == k) continue;
            d[i] -= q[i].re * b[i].re + q[i].im * b[i].im;
#pragma unroll
            for (int j = 0; j < i; ++j) {
                if (j == k) continue;
                l[tri_index(i, j)] = l[tri_index(i, j)] - q[i] * conj(b[j]);
            }
            if (i > k) l[tri_index(i, k)] = q[i];
            else l[tri_index(k, i)] = conj(q[i]);
        }
        d[k] = -r;
    }
#pragma unroll
    for (int k = 0; k < 6; ++k) d[k] = -d[k];
#pragma unroll
    for (int k = 0; k < 15; ++k) l[k] = -l[k];
    return ok;
}

// word pair k of block pb = 2 parity + chirality of half-site h, in the three precisions
LYM_D void store_words(double2 *d, float4 *f, uint2 *hf, size_t stride, int pb, int k, int h, double2 x, double2 y)
{
    const size_t at = (size_t)pb * 9 + k;
    d[at * 2 * stride + h] = x;
    d[(at * 2 + 1) * stride + h] = y;
    f[at * stride + h] = floats(x, y);
    hf[at * stride + h] = halves(x, y);
}

__global__ void __launch_bounds__(128) clover_invert_kernel(CloverArg a)
{
    const int h = blockIdx.x * blockDim.x + threadIdx.x, pb = blockIdx.y;
    if (h >= a.g.Vh) return;
    const size_t st = a.g.stride;
    const double2 *t = a.T + (size_t)pb * 18 * st + h;
    double d[6];
    Cd l[15];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const double2 w = __ldg(t + k * st);
        d[2 * k] = w.x;
        d[2 * k + 1] = w.y;
    }
#pragma unroll
    for (int k = 0; k < 15; ++k) {
        const double2 w = __ldg(t + (3 + k) * st);
        l[k] = Cd{w.x, w.y};
    }
    if (!invert_sweep(d, l)) {
        double2 w[18];
        for (int k = 0; k < 18; ++k) w[k] = __ldg(t + k * st);
        if (!invert_pivoted(w)) atomicOr(a.err, 4);
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            d[2 * k] = w[k].x;
            d[2 * k + 1] = w[k].y;
        }
#pragma unroll
        for (int k = 0; k < 15; ++k) l[k] = Cd{w[3 + k].x, w[3 + k].y};
    }
    auto word = [&](int k) {
        return k < 3 ? make_double2(d[2 * k], d[2 * k + 1]) : make_double2(l[k - 3].re, l[k - 3].im);
    };
#pragma unroll
    for (int k = 0; k < 9; ++k) store_words(a.Ti, a.Tif, a.Tih, st, pb, k, h, word(2 * k), word(2 * k + 1));
}

template <class Gauge> __global__ void __launch_bounds__(kCloverThreads, 2) clover_build_kernel(CloverArg a, Gauge U)
{
    __shared__ __align__(16) double2 sT[2][18][kPad];  // words of T, [chirality][18][site]
    __shared__ double f[6][9][kPad];                   // planes
    const Geom &g = a.g;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int p = blockIdx.y, h = blockIdx.x * kSites + lane;
    const bool in = h < g.Vh;
    int c[4];
    site_coords(g, in ? h : g.Vh - 1, p, c);
    const int mu = warp < 3 ? 0 : (warp < 5 ? 1 : 2), nu = warp < 3 ? warp + 1 : (warp < 5 ? warp - 1 : 3);
    double fl[9];
    plane_of(g, U, c, mu, nu, fl);
#pragma unroll
    for (int e = 0; e < 9; ++e) f[warp][e][lane] = fl[e];
    __syncthreads();
    if (a.F && in) {
        double *o = a.F + ((size_t)lex_of(g, c[0], c[1], c[2], c[3]) * 6 + warp) * 18;
#pragma unroll
        for (int k = 0; k < 9; ++k) {
            const Cd z = plane_entry(f, warp, k % 3, k / 3, lane);
            o[2 * k] = z.re;
            o[2 * k + 1] = z.im;
        }
    }
    {
        // component r = spin * 3 + colour; spins 0, 1 of the block
        const int b = warp / 3, part = warp % 3;
        const double k = b == 0 ? a.kc : -a.kc;
        double2(*t)[kPad] = sT[b];
        auto F = [&](int pl, int i, int j) { return plane_entry(f, pl, i, j, lane); };
        auto put = [&](int w, Cd z) { t[w][lane] = make_double2(z.re, z.im); };
        // the spin-diagonal parts are +-i (F_zt -+ F_xy): sign of a00 is s
        auto diag = [&](int i, int j) { return b == 0 ? F(5, i, j) - F(0, i, j) : F(0, i, j) + F(5, i, j); };
        if (part == 0) {
            double d[6];
#pragma unroll
            for (int i = 0; i < 3; ++i) {
                const double v = k * -diag(i, i).im;
                d[i] = 1.0 + v;
                d[3 + i] = 1.0 - v;
            }
#pragma unroll
            for (int i = 0; i < 3; ++i) t[i][lane] = make_double2(d[2 * i], d[2 * i + 1]);
        }
        if (part != 1) {
            const double s = part == 0 ? k : -k;  // rows and columns 0..2, then 3..5
#pragma unroll
            for (int e = 0; e < 3; ++e) {
                const int i = e == 0 ? 1 : 2, j = e == 2 ? 1 : 0, o = part == 0 ? 0 : 3;
                put(3 + tri_index(o + i, o + j), s * times_i(diag(i, j)));
            }
        } else {
#pragma unroll
            for (int i = 0; i < 3; ++i)
#pragma unroll
                for (int j = 0; j < 3; ++j) {
                    const Cd z = b == 0 ? -F(1, i, j) - F(4, i, j) + times_i(F(2, i, j) - F(3, i, j))
                                        : F(1, i, j) - F(4, i, j) + times_i(F(2, i, j) + F(3, i, j));
                    put(3 + tri_index(3 + i, j), k * z);
                }
        }
    }
    __syncthreads();
    if (!in) return;
    for (int it = warp; it < 18; it += 6) {
        const int b = it / 9, k = it % 9;
        store_words(a.T, a.Tf, a.Th, g.stride, 2 * p + b, k, h, sT[b][2 * k][lane], sT[b][2 * k + 1][lane]);
    }
}

}  // namespace

void launch_store_gauge(const Geom &g, const double *aos, GaugeDev &U, int *err, cudaStream_t st)
{
    const int nb = (g.V + kSites - 1) / kSites;
    if (U.rep == REP_SU3) store_gauge_kernel<double2><<<nb, 128, 0, st>>>(g, (const double2 *)aos, U, err);
    else store_gauge_kernel<double><<<nb, 128, 0, st>>>(g, aos, U, err);
}

void launch_store_gauge8(const Geom &g, GaugeDev &U, cudaStream_t st)
{
    store_gauge8_kernel<<<dim3((g.Vh + 127) / 128, 2, 4), 128, 0, st>>>(g, U);
}

void launch_clover_build(const Geom &g, const GaugeDev &U, double kc, CloverDev &C, double *F_aos, int *err,
                         cudaStream_t st)
{
    const CloverArg a{g,
                      kc,
                      (double2 *)C.T[PREC_D],
                      (double2 *)C.Tinv[PREC_D],
                      (float4 *)C.T[PREC_F],
                      (float4 *)C.Tinv[PREC_F],
                      (uint2 *)C.T[PREC_H],
                      (uint2 *)C.Tinv[PREC_H],
                      F_aos,
                      err};
    const dim3 grid((g.Vh + kSites - 1) / kSites, 2);
    if (U.rep == REP_SU3)
        clover_build_kernel<<<grid, kCloverThreads, 0, st>>>(a, GaugeD18{(const double2 *)U.d64, g.stride});
    else
        clover_build_kernel<<<grid, kCloverThreads, 0, st>>>(a, GaugeD9{(const double *)U.d64, g.stride});
    clover_invert_kernel<<<dim3((g.Vh + 127) / 128, 4), 128, 0, st>>>(a);
}

}  // namespace lym
