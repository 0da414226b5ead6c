// ecg_math.cuh -- register-resident FP64 complex algebra for one ECG pair term.
//
// One pair term is one call of the reference's MatrixElements
// (src/matelem.f90:12-750): bra function k, ket function l acted on by one
// Y^+Y permutation matrix P.  Everything here is n x n with n a template
// parameter (2..5), so every loop unrolls and every matrix lives in
// registers.  All arithmetic is FP64; complex square roots take the
// principal branch exactly as Fortran's intrinsic sqrt does.
#pragma once
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

namespace ecg {

constexpr int NMAX = 5;     // Glob_MaxAllowedNumOfPseudoParticles
constexpr int TMAX = 64;    // largest Y^+Y term count the kernels accept

struct cd {
    double x, y;
};

__host__ __device__ __forceinline__ cd mk(double x, double y) { return cd{x, y}; }
__device__ __forceinline__ cd operator+(cd a, cd b) { return cd{a.x + b.x, a.y + b.y}; }
__device__ __forceinline__ cd operator-(cd a, cd b) { return cd{a.x - b.x, a.y - b.y}; }
__device__ __forceinline__ cd operator-(cd a) { return cd{-a.x, -a.y}; }
__device__ __forceinline__ cd operator*(double s, cd a) { return cd{s * a.x, s * a.y}; }
__device__ __forceinline__ cd operator*(cd a, double s) { return cd{s * a.x, s * a.y}; }
__device__ __forceinline__ cd conj(cd a) { return cd{a.x, -a.y}; }
__device__ __forceinline__ cd cmul(cd a, cd b)
{
    return cd{fma(a.x, b.x, -a.y * b.y), fma(a.x, b.y, a.y * b.x)};
}
__device__ __forceinline__ cd operator*(cd a, cd b) { return cmul(a, b); }
// c + a*b
__device__ __forceinline__ cd cfma(cd a, cd b, cd c)
{
    return cd{fma(a.x, b.x, fma(-a.y, b.y, c.x)), fma(a.x, b.y, fma(a.y, b.x, c.y))};
}
// c - a*b
__device__ __forceinline__ cd cfms(cd a, cd b, cd c)
{
    return cd{fma(-a.x, b.x, fma(a.y, b.y, c.x)), fma(-a.x, b.y, fma(-a.y, b.x, c.y))};
}
// c + s*a, s real
__device__ __forceinline__ cd rfma(double s, cd a, cd c) { return cd{fma(s, a.x, c.x), fma(s, a.y, c.y)}; }
__device__ __forceinline__ double cnorm2(cd a) { return fma(a.x, a.x, a.y * a.y); }
__device__ __forceinline__ cd crcp(cd b)
{
    const double d = 1.0 / cnorm2(b);
    return cd{b.x * d, -b.y * d};
}
// Physical constants of one system: the n x n mass matrix
// Glob_MassMatrix (src/workproc.f90:606-610), pseudo-charges q0, q_i and
// 2^(3n/2) (src/globvars.f90:69).
struct SysParams {
    double M[NMAX * NMAX];  // row-major M[i*NMAX+j]
    double q[NMAX];
    double q0;
    double two_r3n2;
    int n;
    int T;
};

constexpr double SQRTPI = 1.77245385090551602729816748334115;
constexpr double TWO_OVER_SQRTPI = 2.0 / SQRTPI;
constexpr double ONE_OVER_SQRTPI = 1.0 / SQRTPI;

template <int N>
struct Sym {
    static constexpr int NP = N * (N + 1) / 2;
};

// vech index of element (j,i), j >= i, in the column-order vech used by the
// reference (src/matelem.f90:109-122): i outer, j = i..n inner.
__host__ __device__ constexpr int vech_index(int N, int i, int j)
{
    return i * N - i * (i - 1) / 2 + (j - i);
}

// 1/sqrt(x) for positive normal x without a branch: the hardware's seed y
// (rsqrt.approx.ftz.f64), then one step of Householder's method of third
// order, the Taylor series of (1 - e)^(-1/2) to e^2 with e = 1 - x y^2.
// |e| is at most 2^-19.0 over all upper words of the mantissa (measured), so
// the remainder (5/16) e^3 is below 2^-58.  Zero,
// subnormal, infinite or NaN x gives NaN.  rsqrt() and the divide are
// accurate for every x and so end in a branch; the pair term takes up to
// sixteen of them (n = 3), and without the branches their chains overlap.
__device__ __forceinline__ double rsqrt_series(double x)
{
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    const double e = fma(-(x * y), y, 1.0);
    return fma(y * e, fma(0.375, e, 0.5), y);
}
// x clamped to the normal range through its exponent word, x >= 0: what the
// squared modulus of a pivot or a determinant needs where it over- or
// underflows.  (A NaN stays visible in the factor the result multiplies.)
__device__ __forceinline__ double normal_range(double x)
{
    const int hi = min(max(__double2hiint(x), 0x00100000), 0x7fe00000);
    return __hiloint2double(hi, __double2loint(x));
}
// 1/b through the inverse modulus
__device__ __forceinline__ cd crcp_series(cd b)
{
    const double q = rsqrt_series(normal_range(cnorm2(b)));
    const double d = q * q;
    return cd{b.x * d, -b.y * d};
}

// 1/sqrt(a) on the principal branch, and 1/a in ra.  With q = 1/|a| the
// inverse is conj(a) q^2 and its modulus q itself, so Kahan's formulation of
// the square root ("Branch cuts for complex elementary functions", 1987: t =
// sqrt((|x| + |z|)/2), the other component y/(2t)) needs two reciprocal
// square roots and no division.  The branch cut is on the negative real axis,
// as the Fortran intrinsic's.
__device__ __forceinline__ cd crsqrt(cd a, cd& ra)
{
    const double q = rsqrt_series(cnorm2(a));
    const double q2 = q * q;
    ra = cd{a.x * q2, -a.y * q2};
    const double u = 0.5 * (fabs(ra.x) + q);
    const double ri = rsqrt_series(u);
    const double t = u * ri;
    const double h = 0.5 * ra.y * ri;
    const bool pos = ra.x >= 0.0;
    return cd{pos ? t : fabs(h), pos ? h : copysign(t, ra.y)};
}

// The bra data a pair term reads, for one function k: C(i, j) = Ck,
// KM(i, j) = (Ck M)_ij and N6(i, j) = 6 (Ck M Ck)_ij with M the mass matrix.
// BraRegs keeps them in registers (or local memory), BraShared in shared
// memory, entry e of the lane's function at p[e * stride].
template <int N>
struct BraRegs {
    cd c[N][N], km[N][N], n6[N][N];
    __device__ __forceinline__ cd C(int i, int j) const { return c[i][j]; }
    __device__ __forceinline__ cd KM(int i, int j) const { return km[i][j]; }
    __device__ __forceinline__ cd N6(int i, int j) const { return n6[i][j]; }
};
template <int N>
struct BraShared {
    static constexpr int NP = Sym<N>::NP;
    static constexpr int ENTRIES_E = NP + N * N;             // C, KM (energies)
    static constexpr int ENTRIES = 2 * NP + N * N;           // and N6 (gradients)
    const double2* p;
    int stride;
    __device__ __forceinline__ cd at(int e) const
    {
        const double2 v = p[e * stride];
        return cd{v.x, v.y};
    }
    __device__ __forceinline__ cd C(int i, int j) const
    {
        return at(i <= j ? vech_index(N, i, j) : vech_index(N, j, i));
    }
    __device__ __forceinline__ cd KM(int i, int j) const { return at(NP + i * N + j); }
    __device__ __forceinline__ cd N6(int i, int j) const
    {
        return at(NP + N * N + (i <= j ? vech_index(N, i, j) : vech_index(N, j, i)));
    }
};

// X M for symmetric complex X.
template <int N>
__device__ __forceinline__ void mass_right(const cd (&X)[N][N], const SysParams& sp, cd (&XM)[N][N])
{
#pragma unroll
    for (int i = 0; i < N; i++)
#pragma unroll
        for (int j = 0; j < N; j++) {
            cd s = mk(0.0, 0.0);
#pragma unroll
            for (int k = 0; k < N; k++) s = rfma(sp.M[k * NMAX + j], X[i][k], s);
            XM[i][j] = s;
        }
}

// 6 X M X from X and XM = X M.
template <int N>
__device__ __forceinline__ void mass_sandwich(const cd (&X)[N][N], const cd (&XM)[N][N], cd (&N6)[N][N])
{
#pragma unroll
    for (int i = 0; i < N; i++)
#pragma unroll
        for (int j = i; j < N; j++) {
            cd s = mk(0.0, 0.0);
#pragma unroll
            for (int k = 0; k < N; k++) s = cfma(XM[i][k], X[k][j], s);
            N6[i][j] = 6.0 * s;
            N6[j][i] = N6[i][j];
        }
}

// One pair term: what the energy, the derivative and the adjoint kernels
// share.  Inputs: the bra data, tCl = P'A_lP + iP'B_lP (permuted ket),
// absdet = |det L_k det L_l| and scale, a factor on S (2^(3n/2), times the
// term's coefficient and whatever else a caller wants folded in).
//   C = Ck + tCl = L D L^T (unit lower L, no square roots; its pivots are
//   the squares of those of the pseudo-Cholesky factor of
//   src/matelem.f90:203-217, so det C is the same product);
//   X = L^-1 (strict lower part kept), r = 1/D, inv = C^-1 = X^T D^-1 X;
//   S as src/matelem.f90:244-245, times scale;
//   h = H/S: 6 tr[M tCl C^-1 Ck] (src/matelem.f90:248-274), taken as
//   6 sum_k r_k (X Ck M)_k . (X tCl)_k, plus the Coulomb sum
//   (src/matelem.f90:280-299) over S;
//   with GRAD, Qs = Q/sqrt(pi) of ecg_grad.cuh: Q(i,i) = w_ii + sum_{j!=i}
//   w_ij, Q(i,j) = -w_ij, w_ij the Coulomb weights cnumb of
//   src/matelem.f90:677-681 over S.
template <int N>
struct PairTerm {
    cd X[N][N];
    cd r[N];
    cd inv[N][N];
    cd S, h;
    cd Qs[Sym<N>::NP];
};

template <int N, bool GRAD, typename BRA>
__device__ __forceinline__ void pair_term(const BRA& bra, const cd (&tCl)[N][N], double absdet, double scale,
                                          const SysParams& sp, PairTerm<N>& o)
{
    // C = L D L^T by columns: G(j, i) the unscaled column, L(j, i) = G r_i
    cd L[N][N], G[N][N];
    cd det = mk(1.0, 0.0);
#pragma unroll
    for (int i = 0; i < N; i++) {
        cd d = bra.C(i, i) + tCl[i][i];
#pragma unroll
        for (int k = 0; k < i; k++) d = cfms(L[i][k], G[i][k], d);
        det = (i == 0) ? d : det * d;
        o.r[i] = crcp_series(d);
#pragma unroll
        for (int j = i + 1; j < N; j++) {
            cd g = bra.C(i, j) + tCl[i][j];
#pragma unroll
            for (int k = 0; k < i; k++) g = cfms(L[j][k], G[i][k], g);
            G[j][i] = g;
            L[j][i] = cmul(g, o.r[i]);
        }
    }
    // X = L^-1, strict lower
#pragma unroll
    for (int j = 1; j < N; j++)
#pragma unroll
        for (int i = j - 1; i >= 0; i--) {
            cd s = -L[j][i];
#pragma unroll
            for (int k = i + 1; k < j; k++) s = cfms(L[j][k], o.X[k][i], s);
            o.X[j][i] = s;
        }
    // inv = X^T D^-1 X
#pragma unroll
    for (int j = 0; j < N; j++)
#pragma unroll
        for (int i = 0; i <= j; i++) {
            cd s = (i == j) ? o.r[j] : cmul(o.r[j], o.X[j][i]);
#pragma unroll
            for (int k = j + 1; k < N; k++) s = cfma(cmul(o.r[k], o.X[k][j]), o.X[k][i], s);
            o.inv[i][j] = s;
            o.inv[j][i] = s;
        }
    // overlap: c = absdet / det, S = scale c sqrt(c)
    {
        const double q = rsqrt_series(normal_range(cnorm2(det)));
        const double m = absdet * q;  // |c|
        const cd c = cd{m * q * det.x, -m * q * det.y};
        const double u = 0.5 * (fabs(c.x) + m);
        const double ri = rsqrt_series(u);
        const bool pos = c.x >= 0.0, tiny = !(u > 1e-300);  // a vanishing overlap
        const double t = u * ri, hh = 0.5 * c.y * ri;
        const cd sc = tiny ? cd{0.0 * u, 0.0} : cd{pos ? t : fabs(hh), pos ? hh : copysign(t, c.y)};
        o.S = scale * cmul(c, sc);
    }
    // kinetic trace
    cd tr = mk(0.0, 0.0);
#pragma unroll
    for (int k = 0; k < N; k++) {
        cd s = mk(0.0, 0.0);
#pragma unroll
        for (int j = 0; j < N; j++) {
            cd y = bra.KM(k, j), z = tCl[k][j];
#pragma unroll
            for (int a = 0; a < k; a++) {
                y = cfma(o.X[k][a], bra.KM(a, j), y);
                z = cfma(o.X[k][a], tCl[a][j], z);
            }
            s = cfma(y, z, s);
        }
        tr = cfma(o.r[k], s, tr);
    }
    // Coulomb sum over S / (2/sqrt(pi))
    cd v = mk(0.0, 0.0);
    if (GRAD)
#pragma unroll
        for (int i = 0; i < N; i++) o.Qs[vech_index(N, i, i)] = mk(0.0, 0.0);
#pragma unroll
    for (int i = 0; i < N; i++)
#pragma unroll
        for (int j = i; j < N; j++) {
            const cd a = (i == j) ? o.inv[i][i]
                                  : cd{fma(-2.0, o.inv[i][j].x, o.inv[i][i].x + o.inv[j][j].x),
                                       fma(-2.0, o.inv[i][j].y, o.inv[i][i].y + o.inv[j][j].y)};
            cd ra;
            const cd is = crsqrt(a, ra);
            const double qq = (i == j) ? sp.q0 * sp.q[i] : sp.q[i] * sp.q[j];
            v = rfma(qq, is, v);
            if (GRAD) {
                const cd w = (ONE_OVER_SQRTPI * qq) * cmul(is, ra);
                cd& qi = o.Qs[vech_index(N, i, i)];
                qi = qi + w;
                if (i != j) {
                    cd& qj = o.Qs[vech_index(N, j, j)];
                    qj = qj + w;
                    o.Qs[vech_index(N, i, j)] = -w;
                }
            }
        }
    o.h = cd{fma(6.0, tr.x, TWO_OVER_SQRTPI * v.x), fma(6.0, tr.y, TWO_OVER_SQRTPI * v.y)};
}

}  // namespace ecg
