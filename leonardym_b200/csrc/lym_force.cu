// Fermion force of the Wilson and Wilson-clover operators on the device:
// FermionForce::derivative (hmc_forces/FermionForce.cpp:11-20) with the per-link matrices of
// DiracWilsonFermionForce::derivative (hmc_forces/DiracWilsonFermionForce.cpp:10-53) and
// ImprovedFermionForce::derivative (hmc_forces/ImprovedFermionForce.cpp:11-223, the eight
// clover-leaf terms with the link products of its setLattice, :225-268, formed on the fly):
//   force[x][mu] -= weight * F_mu(x),  F = clover / 4 + Wilson.
// X, Y and the force field are in the reference's AoS layout: spinors double2[V][4][3], force
// matrices double2[V][4][3][3] column-major ([site][mu][j][i] = F(i, j)).  Everything in FP64.
//
// Wilson part.  With the half spinors h_k(psi) = psi_k - c_k psi_pk and g_k(psi) = psi_k +
// c_k psi_pk of direction mu (the projections of lym_dslash.cuh), the sum over the spins and
// both pair orders of the first term is
//   M = sum_i w_i sum_{k=0,1} h_k(Y_i)(x+mu) g_k(X_i)(x)^+ + h_k(X_i)(x+mu) g_k(Y_i)(x)^+ ,
// the second term's spin sum is M^+, and F = -kappa (M - (U M U)^+) with U = U_mu(x): the link
// enters once per (site, mu), not once per pair and spin.
//
// Clover part.  gamma5 sigma_{mu nu} acts inside a chirality as +- a Pauli matrix, so the six
// plane matrices N^{mu nu}(x) of the spinors are i times real combinations of the Hermitian
//   P_k = sum_ab (sigma_k)_ab sum_i w_i (Y_b X_a^+ + X_b Y_a^+)   (k = 1..3, per chirality),
// 9 reals each (H below, kappa c_sw and the signs included).  The eight terms of a plane are
//   i [H(x+mu) V + V H(x) + C S] for the staple V = C E through x+nu, and minus the adjoint of
// the same expression through x-nu between two U_mu(x)^+, with E = B^+ A^+, C = U_nu(x+mu),
// B = U_mu(x+nu), A = U_nu(x), S = H(x+mu+nu) E + B^+ (H(x+nu) A^+): 8 matrix products per
// staple, two of them with a packed Hermitian factor.
#include "lym_common.cuh"
#include "lym_dslash.cuh"
#include "lym_internal.h"
#include "lym_mat3.cuh"

namespace lym {

namespace {

typedef Cd C;

// a Hermitian matrix: 3 diagonal reals, entries (0,1), (0,2), (1,2)
struct Herm {
    double d[3];
    C o[3];
    LYM_D C at(int i, int j) const  // i != j
    {
        return i < j ? o[i + j - 1] : lym::conj(o[i + j - 1]);
    }
};
// R += H B, R += A H
template <class T> LYM_D void mul_add(Mat<C> &R, const Herm &H, const Mat<T> &B)
{
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int j = 0; j < 3; ++j)
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                if (k == i) acc(R.a[i][j], H.d[i], B.a[k][j]);
                else acc(R.a[i][j], H.at(i, k), B.a[k][j]);
            }
}
template <class T> LYM_D void mul_add(Mat<C> &R, const Mat<T> &A, const Herm &H)
{
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int j = 0; j < 3; ++j)
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                if (k == j) acc(R.a[i][j], A.a[i][k], H.d[j]);
                else acc(R.a[i][j], A.a[i][k], H.at(k, j));
            }
}
// F(i, j) += y_i conj(x_j)  (FermionForce.cpp:22-31)
LYM_D void add_outer(Mat<C> &F, const C y[3], const C x[3])
{
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int j = 0; j < 3; ++j) fma_cc(F.a[i][j], x[j], y[i]);
}

struct ForceArg {
    Geom g;
    int n;                     // pairs (x_i, y_i) with weights w_i
    const double2 *const *X;   // device array [n] of AoS spinors
    const double2 *const *Y;
    const double *w;           // device array [n]
    double2 *force;
    double *N;  // plane matrices H [parity][plane][9][stride] (clover only)
    double kappa, csw;
    int clover;
};

// force -= F at the AoS matrix `out`
LYM_D void subtract(double2 *out, const Mat<C> &F)
{
#pragma unroll
    for (int j = 0; j < 3; ++j)
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            double2 w = out[j * 3 + i];
            w.x -= F.a[i][j].re;
            w.y -= F.a[i][j].im;
            out[j * 3 + i] = w;
        }
}

// ---------------------------------------------------------------- spinors --
// One block takes 32 consecutive sites (lexicographic).  Per pair it copies X and Y of these
// sites and of their forward neighbours into shared memory (12 16-byte words a site, so the
// copies are contiguous 192-byte pieces); warps 0..3 then add the pair to M of direction mu =
// warp, warps 4 and 5 to the P_k of one chirality (27 reals a thread).  The +t neighbour of a
// site is the next site of the tile, except at the end of a t line or of the tile: only those
// are copied for it.  Bound by shared memory traffic (8 x 192 bytes written and 36 x 96 read per
// site and pair: L1 and shared memory at half of their rate, DRAM at 43 %, FP64 at 22 %) and its
// latency at 12 warps per SM, so the next pair's copies run during this pair's sums, two blocks
// per SM; the
// order of the tiles (x slowest, or columns that keep the +x neighbours in L2) made no
// difference.  Reading the AoS spinors straight into registers instead costs one 32-byte sector
// per lane and load, with 48 loads per pair, site and direction.
// 24^3 x 48, 12 pairs: 2.16 ms (2.40 with one stage and all +t neighbours copied), against
// 3.8 ms for six plane matrices per site plus most of 18.9 ms for the Wilson part per pair.
constexpr int kTile = 32;
constexpr int kVecWords = 13;                   // 12 words of a spinor, 1 of padding: conflict-free reads
constexpr int kRun = kTile * kVecWords;         // words of one vector of the tile
constexpr int kSpinThreads = 192;
// X or Y of one pair: own, +x, +y, +z sites, then the extra +t sites
LYM_HD int extra_t_sites(int Lt) { return (Lt - 1 + kTile - 1) / Lt + 1; }
LYM_HD int vector_words(int Lt) { return 4 * kRun + extra_t_sites(Lt) * kVecWords; }
inline int spin_smem(int Lt) { return 2 * 2 * vector_words(Lt) * 16; }  // two stages of X and Y

LYM_D void copy16(double2 *dst, const double2 *src)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"((unsigned)__cvta_generic_to_shared(dst)),
                 "l"(src)
                 : "memory");
}

template <int S> LYM_D void half_spinor(const double2 *v, int mu, int k, C o[3])  // psi_k + S c_k psi_pk
{
    const int pk = proj_partner(mu, k), code = proj_code(mu, k);
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        const double2 a = v[3 * k + d], b = v[3 * pk + d];
        const C z = mul_code(code, C{b.x, b.y});
        o[d] = S > 0 ? C{a.x, a.y} + z : C{a.x, a.y} - z;
    }
}

// x0: X of the site, xf: X of its +mu neighbour; yo: words from X to Y
template <int MU> LYM_D void add_wilson(const double2 *x0, const double2 *xf, int yo, double w, Mat<C> &M)
{
    const double2 *y0 = x0 + yo, *yf = xf + yo;
#pragma unroll
    for (int k = 0; k < 2; ++k)
#pragma unroll
        for (int o = 0; o < 2; ++o) {
            C h[3], g[3];
            half_spinor<-1>(o ? xf : yf, MU, k, h);
            half_spinor<+1>(o ? y0 : x0, MU, k, g);
#pragma unroll
            for (int d = 0; d < 3; ++d) h[d] = w * h[d];
            add_outer(M, h, g);
        }
}

template <class Gauge, bool CLOVER>
__global__ void __launch_bounds__(kSpinThreads, 2) spinor_force_kernel(ForceArg a, Gauge U)
{
    extern __shared__ __align__(16) double2 sm[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int s0 = blockIdx.x * kTile;
    const int V = a.g.V, Lt = a.g.L[3];
    const int yo = vector_words(Lt), t0 = s0 % Lt;
    // the copies of this thread: word w of the sites j0 and j0 + 16, own and neighbours
    const int j0 = threadIdx.x / 12, w = threadIdx.x % 12;
    int src[2][5], slot[2];
#pragma unroll
    for (int q = 0; q < 2; ++q) {
        const int j = j0 + 16 * q;
        const int s = min(s0 + j, V - 1);
        int c[4];
        coords_of(a.g, s, c);
        src[q][0] = s;
#pragma unroll
        for (int mu = 0; mu < 4; ++mu) {
            int o[4];
            moved(a.g, c, mu, +1, o);
            src[q][1 + mu] = lex_of(a.g, o[0], o[1], o[2], o[3]);
        }
        slot[q] = (c[3] == Lt - 1 || j == kTile - 1) ? (t0 + j) / Lt : -1;
    }
    auto copy_pair = [&](int i, int stage) {
        const double2 *X = a.X[i] + w, *Y = a.Y[i] + w;
        double2 *base = sm + stage * 2 * yo + w;
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            double2 *d = base + (j0 + 16 * q) * kVecWords;
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                copy16(d + r * kRun, X + (size_t)src[q][r] * 12);
                copy16(d + yo + r * kRun, Y + (size_t)src[q][r] * 12);
            }
            if (slot[q] >= 0) {
                double2 *e = base + 4 * kRun + slot[q] * kVecWords;
                copy16(e, X + (size_t)src[q][4] * 12);
                copy16(e + yo, Y + (size_t)src[q][4] * 12);
            }
        }
        asm volatile("cp.async.commit_group;\n" ::: "memory");
    };
    const bool t_end = (t0 + lane) % Lt == Lt - 1 || lane == kTile - 1;
    const int t_word = t_end ? 4 * kRun + (t0 + lane) / Lt * kVecWords : (lane + 1) * kVecWords;
    Mat<C> M;  // warps 0..3
    zero(M);
    double P[27];  // warps 4, 5: M_01 (18), M_00 - M_11 (9, Hermitian)
#pragma unroll
    for (int k = 0; k < 27; ++k) P[k] = 0.0;
    copy_pair(0, 0);
#pragma unroll 1
    for (int i = 0; i < a.n; ++i) {
        if (i + 1 < a.n) {
            copy_pair(i + 1, (i + 1) & 1);
            asm volatile("cp.async.wait_group 1;\n" ::: "memory");
        } else {
            asm volatile("cp.async.wait_group 0;\n" ::: "memory");
        }
        __syncthreads();
        const double2 *st = sm + (i & 1) * 2 * yo, *own = st + lane * kVecWords;
        const double wi = a.w[i];
        switch (warp) {
        case 0: add_wilson<0>(own, own + 1 * kRun, yo, wi, M); break;
        case 1: add_wilson<1>(own, own + 2 * kRun, yo, wi, M); break;
        case 2: add_wilson<2>(own, own + 3 * kRun, yo, wi, M); break;
        case 3: add_wilson<3>(own, st + t_word, yo, wi, M); break;
        default:
            if constexpr (CLOVER) {
                const double2 *x = own + (warp - 4) * 6, *y = x + yo;
                C x0[3], x1[3], y0[3], y1[3];
#pragma unroll
                for (int d = 0; d < 3; ++d) {
                    x0[d] = wi * C{x[d].x, x[d].y};
                    x1[d] = wi * C{x[3 + d].x, x[3 + d].y};
                    y0[d] = C{y[d].x, y[d].y};
                    y1[d] = C{y[3 + d].x, y[3 + d].y};
                }
                // M_ab(i, j) = y_b,i conj(x_a,j) + x_b,i conj(y_a,j)
#pragma unroll
                for (int r = 0; r < 3; ++r)
#pragma unroll
                    for (int q = 0; q < 3; ++q) {
                        C t{P[2 * (3 * r + q)], P[2 * (3 * r + q) + 1]};
                        fma_cc(t, x0[q], y1[r]);
                        fma_cc(t, y0[q], x1[r]);
                        P[2 * (3 * r + q)] = t.re;
                        P[2 * (3 * r + q) + 1] = t.im;
                    }
#pragma unroll
                for (int r = 0; r < 3; ++r)
                    P[18 + r] += 2.0 * ((y0[r].re * x0[r].re + y0[r].im * x0[r].im) -
                                        (y1[r].re * x1[r].re + y1[r].im * x1[r].im));
#pragma unroll
                for (int e = 0; e < 3; ++e) {
                    const int r = e == 2 ? 1 : 0, q = e == 0 ? 1 : 2;
                    C t{P[21 + 2 * e], P[22 + 2 * e]};
                    fma_cc(t, x0[q], y0[r]);
                    fma_cc(t, y0[q], x0[r]);
                    fma_cc(t, -x1[q], y1[r]);
                    fma_cc(t, -y1[q], x1[r]);
                    P[21 + 2 * e] = t.re;
                    P[22 + 2 * e] = t.im;
                }
            }
        }
        __syncthreads();  // before a later pair's copies land on these
    }
    const int s = s0 + lane;
    if (warp < 4) {
        if (s < V) {
            int c[4];
            coords_of(a.g, s, c);
            const Site own = site_of(a.g, c);
            const auto Um = load_link(U, own.p, warp, own.h);
            const Mat<C> UMU = mul(mul(Um, M), Um);
#pragma unroll
            for (int i = 0; i < 3; ++i)
#pragma unroll
                for (int j = 0; j < 3; ++j) M.a[i][j] = (-a.kappa) * (M.a[i][j] - lym::conj(UMU.a[j][i]));
            subtract(a.force + ((size_t)s * 4 + warp) * 9, M);
        }
    }
    if constexpr (CLOVER) {
        // the P_k of both chiralities, then H = kappa c_sw (su P_k(upper) + sl P_k(lower)):
        // planes 03, 13, 23 (k = x, y, z): su = sl = 1; 12, 02, 01: su = -e, sl = e, e = 1, -1, 1
        double *ex = reinterpret_cast<double *>(sm);  // [chirality][27][33]
        if (warp >= 4) {
#pragma unroll
            for (int k = 0; k < 27; ++k) ex[((warp - 4) * 27 + k) * 33 + lane] = P[k];
        }
        __syncthreads();
        if (warp < 3 && s < V) {
            const int k = warp;  // Pauli index; this warp writes its space and its time plane
            int c[4];
            coords_of(a.g, s, c);
            const Site own = site_of(a.g, c);
            double h[2][9];
#pragma unroll
            for (int b = 0; b < 2; ++b) {
                const double *m = ex + b * 27 * 33 + lane;
                if (k == 2) {
#pragma unroll
                    for (int e = 0; e < 9; ++e) h[b][e] = m[(18 + e) * 33];
                } else {
                    // P_1 = M_01 + M_01^+, P_2 = -i (M_01 - M_01^+)
#pragma unroll
                    for (int r = 0; r < 3; ++r) h[b][r] = 2.0 * m[(8 * r + k) * 33];
#pragma unroll
                    for (int e = 0; e < 3; ++e) {
                        const int r = e == 2 ? 1 : 0, q = e == 0 ? 1 : 2;
                        const double ur = m[2 * (3 * r + q) * 33], ui = m[(2 * (3 * r + q) + 1) * 33];
                        const double lr = m[2 * (3 * q + r) * 33], li = m[(2 * (3 * q + r) + 1) * 33];
                        h[b][3 + 2 * e] = k == 0 ? ur + lr : ui + li;
                        h[b][4 + 2 * e] = k == 0 ? ui - li : lr - ur;
                    }
                }
            }
            const double kc = a.kappa * a.csw, sp = k == 1 ? kc : -kc;
            const int space = k == 0 ? 3 : (k == 1 ? 1 : 0), time = k == 0 ? 2 : (k == 1 ? 4 : 5);
            double *ns = a.N + (size_t)((own.p * 6 + space) * 9) * a.g.stride + own.h;
            double *nt = a.N + (size_t)((own.p * 6 + time) * 9) * a.g.stride + own.h;
#pragma unroll
            for (int e = 0; e < 9; ++e) {
                ns[(size_t)e * a.g.stride] = sp * (h[0][e] - h[1][e]);
                nt[(size_t)e * a.g.stride] = kc * (h[0][e] + h[1][e]);
            }
        }
    }
}

// ----------------------------------------------------------------- clover --
// planes (mu < nu): 01 02 03 12 13 23
LYM_D int plane_index(int mu, int nu)
{
    const int a = mu < nu ? mu : nu, b = mu < nu ? nu : mu;
    return a == 0 ? b - 1 : (a == 1 ? b + 1 : 5);
}
LYM_D Herm load_plane(const ForceArg &a, Site s, int plane)
{
    const double *b = a.N + (size_t)((s.p * 6 + plane) * 9) * a.g.stride + s.h;
    double v[9];
#pragma unroll
    for (int e = 0; e < 9; ++e) v[e] = __ldg(b + (size_t)e * a.g.stride);
    Herm H;
#pragma unroll
    for (int e = 0; e < 3; ++e) {
        H.d[e] = v[e];
        H.o[e] = C{v[3 + 2 * e], v[4 + 2 * e]};
    }
    return H;
}

// acc += sgn (H(x+mu) V + V H(x) + C S), the staple V = C E of plane (mu, nu) through x + nu
// (UP) or x - nu, with A+ = U_nu(x)^+ or U_nu(x-nu) and C = U_nu(x+mu) or U_nu(x+mu-nu)^+
template <bool UP, class Gauge>
LYM_D void add_staple(const ForceArg &a, const Gauge &U, const int c[4], const int cm[4], int mu, int nu, double sgn,
                      Mat<C> &F)
{
    const Geom &g = a.g;
    const int plane = plane_index(mu, nu);
    int o[4];
    const Site x = site_of(g, c), xm = site_of(g, cm);
    moved(g, c, nu, UP ? +1 : -1, o);
    const Site xn = site_of(g, o);
    moved(g, cm, nu, UP ? +1 : -1, o);
    const Site xmn = site_of(g, o);
    const auto Al = load_link(U, UP ? x.p : xn.p, nu, UP ? x.h : xn.h);
    const auto A = UP ? dag(Al) : Al;
    Mat<C> K;  // H(x+-nu) A + A H(x)
    zero(K);
    mul_add(K, load_plane(a, xn, plane), A);
    mul_add(K, A, load_plane(a, x, plane));
    const auto B = dag(load_link(U, xn.p, mu, xn.h));
    Mat<C> S = mul(B, K);
    const auto E = mul(B, A);
    mul_add(S, load_plane(a, xmn, plane), E);
    const auto Cl = load_link(U, UP ? xm.p : xmn.p, nu, UP ? xm.h : xmn.h);
    const auto Cc = UP ? Cl : dag(Cl);
    Mat<C> T = mul(Cc, S);
    mul_add(T, load_plane(a, xm, plane), mul(Cc, E));
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int j = 0; j < 3; ++j) fma_r(F.a[i][j], sgn, T.a[i][j]);
}

// One thread per (half-site, mu); a block's four warps take the four directions of 32
// consecutive half-sites, whose links and plane matrices they share through L1.  Bound by FP64
// arithmetic (about 20k fused multiply-adds per site, 0.8 ms of the chip at 24^3 x 48; the FP64 pipe
// is busy half of the time with 8 warps per SM), so it runs at 252 registers, two blocks per SM,
// rather than spill: 1.51 ms there (11 link products
// and 10 with plane matrices per staple pair before, most of 18.9 ms).  The lower staples come
// first: their sum L enters as -(U L U)^+.
template <class Gauge> __global__ void __launch_bounds__(128, 2) clover_force_kernel(ForceArg a, Gauge U)
{
    const int h = blockIdx.x * 32 + (threadIdx.x & 31), p = blockIdx.y, mu = threadIdx.x >> 5;
    if (h >= a.g.Vh) return;
    int c[4], cm[4];
    site_coords(a.g, h, p, c);
    moved(a.g, c, mu, +1, cm);
    Mat<C> F;
    zero(F);
#pragma unroll 1
    for (int nu = 0; nu < 4; ++nu)
        if (nu != mu) add_staple<false>(a, U, c, cm, mu, nu, mu < nu ? 1.0 : -1.0, F);
    {
        const auto Um = load_link(U, p, mu, h);
        F = mul(mul(Um, F), Um);
        F = dag(F);
#pragma unroll
        for (int i = 0; i < 3; ++i)
#pragma unroll
            for (int j = 0; j < 3; ++j) F.a[i][j] = -F.a[i][j];
    }
#pragma unroll 1
    for (int nu = 0; nu < 4; ++nu)
        if (nu != mu) add_staple<true>(a, U, c, cm, mu, nu, mu < nu ? 1.0 : -1.0, F);
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int j = 0; j < 3; ++j) F.a[i][j] = 0.25 * times_i(F.a[i][j]);
    subtract(a.force + ((size_t)lex_of(a.g, c[0], c[1], c[2], c[3]) * 4 + mu) * 9, F);
}

template <class Gauge, bool CLOVER> void run_spinor_force(const ForceArg &a, const Gauge &U, cudaStream_t st)
{
    const int smem = spin_smem(a.g.L[3]);
    cudaFuncSetAttribute(spinor_force_kernel<Gauge, CLOVER>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    spinor_force_kernel<Gauge, CLOVER><<<(a.g.V + kTile - 1) / kTile, kSpinThreads, smem, st>>>(a, U);
}

template <class Gauge> void run_force(const ForceArg &a, const Gauge &U, cudaStream_t st)
{
    if (a.clover) {
        run_spinor_force<Gauge, true>(a, U, st);
        clover_force_kernel<Gauge><<<dim3((a.g.Vh + 31) / 32, 2), 128, 0, st>>>(a, U);
    } else {
        run_spinor_force<Gauge, false>(a, U, st);
    }
}

}  // namespace

size_t fermion_force_scratch_bytes(const Geom &g) { return (size_t)2 * 6 * 9 * g.stride * sizeof(double); }

void launch_fermion_force(const Geom &g, const GaugeDev &U, int n, const double2 *const *X, const double2 *const *Y,
                          const double *weights, double kappa, double csw, int clover, double2 *force,
                          double *scratch, cudaStream_t st)
{
    const ForceArg a{g, n, X, Y, weights, force, scratch, kappa, csw, clover};
    if (U.rep == REP_SU3) run_force(a, GaugeD18{(const double2 *)U.d64, g.stride}, st);
    else run_force(a, GaugeD9{(const double *)U.d64, g.stride}, st);
}

}  // namespace lym
