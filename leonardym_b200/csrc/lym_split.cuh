// The FP64 Wilson-clover stencil: four threads per site.
//
// Thread (k, d) of a site, k, d = 0, 1, takes the half spinor h_k (lym_dslash.cuh) of the
// directions mu = 2 d, 2 d + 1: it accumulates upper spin k and the lower spin its two
// directions pair with k (3 - k for d = 0, 2 + k for d = 1), 6 complex numbers instead of the 12
// of a thread per site, then the lanes of the site add up their parts by shuffles:
//   spin k      = up(k, 0) + up(k, 1),   spin 2 + k = low(k, 1) + low(1 - k, 0),
// after which thread (k, d) holds spin 2 d + k and applies its three rows of the clover block of
// chirality d.  A warp is 8 sites, lane = site + 8 d + 16 k, so that link loads of k = 0, 1 fall
// on one address and spinor loads on contiguous 128-byte pieces.
//
// Why four threads: in FP64 the whole-site form needs 142-180 registers (3 blocks of 128 per SM,
// 12 warps), too few loads in flight for HBM, and on small lattices too few warps and one long
// dependent chain per site.  24^3 x 48: both parities in one launch 247 us against
// 2 x 144 us, one parity 141-149 against 144 us (T^-1 half 130 against 137); 16^3 x 32 adjoint 25
// and 21 against 26 and 28 us; 8^4 both parities 4.6 against 2 x 6.6 us.  Latency bound (L1 misses;
// 4.35 TB/s of HBM, 16 warps per SM): 3, 5 or 6 blocks per SM give 253, 270, 312 us there, blocks
// of 256 or 512 threads 252, 280 us.
#pragma once

#include "lym_common.cuh"
#include "lym_dslash.cuh"

namespace lym {
namespace split {

typedef cx<double> C;

constexpr int kSplitThreads = 128;
constexpr int kSplitSites = kSplitThreads / 4;

LYM_D C load1(const SpinorD &v, int word, int h)
{
    const double2 w = __ldg(v.v + (size_t)word * v.stride + h);
    return C{w.x, w.y};
}
LYM_D C shfl_xor(C z, int m)
{
    return C{__shfl_xor_sync(0xffffffffu, z.re, m), __shfl_xor_sync(0xffffffffu, z.im, m)};
}

// spin 2 d + k of H x at the site (p, h), lexicographic index s, coordinates c; load(w, sn) gives
// word w of x at the site of lexicographic index sn, on the other parity
template <class Load, class GaugeT>
LYM_D void split_hopping(const Geom &g, const Load &load, const GaugeT &U, int p, int h, int s, const int c[4], int k,
                         int d, C own[3])
{
    C up[3], low[3];
#pragma unroll
    for (int m = 0; m < 3; ++m) up[m] = low[m] = C{0.0, 0.0};
    const int wk = 3 * k, wp = 3 * (d ? 2 + k : 3 - k);
#pragma unroll
    for (int j = 0; j < 2; ++j) {
        const int mu = 2 * d + j;
        const int cm = d ? c[2 + j] : c[j], L = d ? g.L[2 + j] : g.L[j];
        const int step = j == 0 ? (d ? g.L[3] : g.L[1] * g.L[2] * g.L[3]) : (d ? 1 : g.L[2] * g.L[3]);
        // c_mu = -i s (j = 0) or s (j = 1)
        const double sg = j == 0 ? (d & k ? -1.0 : 1.0) : (d | k ? 1.0 : -1.0);
#pragma unroll
        for (int dir = 0; dir < 2; ++dir) {
            const int sn = s + (dir == 0 ? (cm == L - 1 ? (1 - L) * step : step) : (cm == 0 ? (L - 1) * step : -step));
            const double sh = dir == 0 ? -sg : sg;
            typename GaugeT::Link Lk;
            if (dir == 0) U.load(p, mu, h, Lk);
            else U.load(1 - p, mu, sn >> 1, Lk);
            C hv[3], w[3];
#pragma unroll
            for (int m = 0; m < 3; ++m) {
                const C xk = load(wk + m, sn), xp = load(wp + m, sn);
                const C z = j == 0 ? times_mi(xp) : xp;
                hv[m] = xk;
                fma_r(hv[m], sh, z);
            }
            if (dir == 0) mul_u(Lk, hv, w);
            else mul_ud(Lk, hv, w);
#pragma unroll
            for (int m = 0; m < 3; ++m) {
                up[m] = up[m] + w[m];
                fma_r(low[m], sh, j == 0 ? times_i(w[m]) : w[m]);
            }
        }
    }
#pragma unroll
    for (int m = 0; m < 3; ++m) {
        up[m] = up[m] + shfl_xor(up[m], 8);
        low[m] = low[m] + shfl_xor(low[m], 24);
        own[m] = d ? low[m] : up[m];
    }
}

// The clover words of a thread in its own shared-memory slots (word w at [w][thread]): the
// diagonal's two words, the three below the diagonal inside the own spin, the nine entries (own
// spin row i, other spin column j) of the block or, for k = 0, of its transpose.  The one-launch CG
// keeps them there; fetching them (and y) ahead of the hopping term in the launches of
// lym_split.cu took L1 from the stencil and was slower (252 against 247 us at 24^3 x 48).
constexpr int kCloverWords = 14;

LYM_D void copy16(double2 *dst, const double2 *src)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"((unsigned)__cvta_generic_to_shared(dst)),
                 "l"(src)
                 : "memory");
}
// the place in the block (parity p, chirality d) of word w of thread k's slots
LYM_D int clover_word(int w, int k)
{
    if (w < 2) return w == 0 ? 1 : (k ? 2 : 0);
    if (w < 5) return 3 + (w == 2 ? (k ? 9 : 0) : w == 3 ? (k ? 13 : 1) : (k ? 14 : 2));
    // word of (3 + i, 0): 3 + tri_index(3 + i, 0) = 6, 9, 13
    const int i = (w - 5) / 3, j = (w - 5) % 3;
    const int ri = i == 0 ? 6 : i == 1 ? 9 : 13, rj = j == 0 ? 6 : j == 1 ? 9 : 13;
    return k ? ri + j : rj + i;
}
LYM_D void fetch_clover(double2 *own, const double2 *clover, int stride, int p, int h, int k, int d)
{
    const double2 *base = clover + (size_t)((p * 2 + d) * 18) * stride + h;
#pragma unroll
    for (int w = 0; w < kCloverWords; ++w) copy16(own + w * kSplitThreads, base + (size_t)clover_word(w, k) * stride);
}
// rows 3 k .. 3 k + 2 of the Hermitian 6 x 6 block (chirality d) applied to the vector (own spin k,
// other spin 1 - k); word(w) gives word w of the thread's slots
template <class Word> LYM_D void clover_rows(const Word &word, int k, const C own[3], const C oth[3], C res[3])
{
    auto entry = [&](int w) {
        const double2 z = word(w);
        return C{z.x, z.y};
    };
    const C dm = entry(0), de = entry(1);
    const double dg[3] = {k ? dm.im : de.re, k ? de.re : de.im, k ? de.im : dm.re};
#pragma unroll
    for (int i = 0; i < 3; ++i) res[i] = dg[i] * own[i];
    const C o10 = entry(2), o20 = entry(3), o21 = entry(4);
    fma_cc(res[0], o10, own[1]);
    fma_c(res[1], o10, own[0]);
    fma_cc(res[0], o20, own[2]);
    fma_c(res[2], o20, own[0]);
    fma_cc(res[1], o21, own[2]);
    fma_c(res[2], o21, own[1]);
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int j = 0; j < 3; ++j) {
            const C e = entry(5 + 3 * i + j);
            fma_c(res[i], C{e.re, k ? e.im : -e.im}, oth[j]);
        }
}

}  // namespace split
}  // namespace lym
