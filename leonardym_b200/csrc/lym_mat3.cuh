// 3x3 FP64 colour matrices, complex (SU(3)) or real (adjoint SU(2)) by element type, and the
// site arithmetic of the kernels that walk loops of links (fermion force, clover term).
#pragma once

#include "lym_common.cuh"

namespace lym {

typedef cx<double> Cd;

template <class T> struct Mat {
    T a[3][3];  // a[i][j] = M(i, j)
};

// r += a b over real and complex factors (adjoint links are real)
LYM_D void acc(Cd &r, Cd a, Cd b) { fma_c(r, a, b); }
LYM_D void acc(Cd &r, double a, Cd b) { fma_r(r, a, b); }
LYM_D void acc(Cd &r, Cd a, double b) { fma_r(r, b, a); }
LYM_D void acc(Cd &r, double a, double b) { r.re = fma(a, b, r.re); }
LYM_D void acc(double &r, double a, double b) { r = fma(a, b, r); }
LYM_D double conj(double a) { return a; }
LYM_D void zero(Cd &a) { a = Cd{0.0, 0.0}; }
LYM_D void zero(double &a) { a = 0.0; }

template <class A, class B> struct Prod {
    typedef Cd T;
};
template <> struct Prod<double, double> {
    typedef double T;
};

template <class T> LYM_D Mat<T> dag(const Mat<T> &A)
{
    Mat<T> R;
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int j = 0; j < 3; ++j) R.a[i][j] = conj(A.a[j][i]);
    return R;
}
template <class TR, class TA, class TB> LYM_D void mul_add(Mat<TR> &R, const Mat<TA> &A, const Mat<TB> &B)
{
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int j = 0; j < 3; ++j)
#pragma unroll
            for (int k = 0; k < 3; ++k) acc(R.a[i][j], A.a[i][k], B.a[k][j]);
}
template <class TA, class TB>
LYM_D Mat<typename Prod<TA, TB>::T> mul(const Mat<TA> &A, const Mat<TB> &B)
{
    Mat<typename Prod<TA, TB>::T> R;
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int j = 0; j < 3; ++j) zero(R.a[i][j]);
    mul_add(R, A, B);
    return R;
}
template <class T> LYM_D void zero(Mat<T> &M)
{
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int j = 0; j < 3; ++j) zero(M.a[i][j]);
}

template <class T> struct LinkOf;
template <> struct LinkOf<GaugeD18> {
    typedef Cd T;
};
template <> struct LinkOf<GaugeD9> {
    typedef double T;
};
template <class Gauge> LYM_D Mat<typename LinkOf<Gauge>::T> load_link(const Gauge &U, int p, int mu, int h)
{
    typename Gauge::Link L;
    U.load(p, mu, h, L);
    Mat<typename LinkOf<Gauge>::T> M;
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int j = 0; j < 3; ++j) M.a[i][j] = L.u[i][j];
    return M;
}

// a site by its coordinates: parity and half-site index
struct Site {
    int p, h;
};
LYM_D Site site_of(const Geom &g, const int c[4])
{
    return Site{(c[0] + c[1] + c[2] + c[3]) & 1, lex_of(g, c[0], c[1], c[2], c[3]) >> 1};
}
LYM_D void coords_of(const Geom &g, int s, int c[4])
{
    c[3] = s % g.L[3];
    int r = s / g.L[3];
    c[2] = r % g.L[2];
    r /= g.L[2];
    c[1] = r % g.L[1];
    c[0] = r / g.L[1];
}
// c moved by d in direction mu (periodic); mu is not a compile-time constant
LYM_D void moved(const Geom &g, const int c[4], int mu, int d, int o[4])
{
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        int v = c[k];
        if (k == mu) {
            v += d;
            if (v >= g.L[k]) v -= g.L[k];
            if (v < 0) v += g.L[k];
        }
        o[k] = v;
    }
}

}  // namespace lym
