// expc.cu -- expectation values over an eigenvector: the pair terms of
// MatrixElementsForExpcVals (src/matelem.f90:949-1983) and the weighted
// sums of ExpectationValuesG's main loop (src/workproc.f90:8159-8366).
//
// One thread evaluates one pair (row i >= column j) for every symmetry term
// of the list, and adds each value's weight  factor * coef * Re(c_i^* c_j O)
// and its rounding-error bound (the reference's MEkl_s / MEkl_e) to sums over
// its warp as the value is produced, so no pair term is stored.  A second
// kernel sums the blocks; every order is fixed, so the result does not
// depend on scheduling.  Correlation functions and particle densities
// (the grid parts) run as a second pair kernel whose blocks also split the
// grid, with the same two-level reduction.
//
// The n x n algebra is restated through three matrices.  With C = tCk + tCl,
// a pair index P = (a, b), u_P = e_a (a = b) or e_a - e_b and TrCJ_P =
// u_P' C^-1 u_P, the traces of ME_rXr_over_rij, ME_rXr_rYr_over_rij, ME_dXd
// and ME_dXd_dYd (src/matelem.f90:753-945) are quadratic forms in C^-1 tCl,
// C^-1 tCk and X = tCk C^-1 tCl, and tCk C^-1 tCk = tCk - X, tCl C^-1 tCl =
// tCl - X (all symmetric).  Put in, the long sums the reference takes term
// by term leave
//   kinetic            6 S tr[M X]
//   mass-velocity      -(36/8) (5/3) S ((sum of all X_kl)^2 / m0^3 + sum_i X_ii^2 / m_i^3)
//   ME_dXd_dYd         36 X_ii X_jj + 24 X_ij^2 (X = E_ii, Y = E_jj)
//   orbit-orbit        -8 X_ij <1/r_P> of each (i, j)
// so the Drachmanised mass-velocity and Darwin sums are one value (the
// reference's own check of them), and the cancellation between the terms,
// which cost the orbit-orbit term up to seven digits, does not happen.
// Results agree with the reference's to its rounding.
//
// TrCJCJ(i,j,p,q) of src/matelem.f90:1270-1300 is never assigned for
// i = j < p < q (n >= 3) but is read by the 1/(r_ij r_pq) loop; the
// reference's ifort build keeps local arrays in zero-initialised static
// storage, so those entries are zero there.  k_expc takes zero for them too.
#include <float.h>
#include <algorithm>
#include "ecg_internal.h"
#include "warp_sums.cuh"

namespace ecg {

namespace {

constexpr int EXPC_BLK = 128;
constexpr int EXPC_MINB = 2;  // CTAs an SM
constexpr int GRID_BLK = 64;
constexpr double PI_D = 3.14159265358979323846264338327950;

__device__ __forceinline__ cd cexp_(cd z)
{
    double s, c;
    sincos(z.y, &s, &c);
    const double e = exp(z.x);
    return mk(e * c, e * s);
}

template <int N>
__device__ __forceinline__ void mm(const cd (&A)[N][N], const cd (&B)[N][N], cd (&C)[N][N])
{
#pragma unroll
    for (int i = 0; i < N; i++)
#pragma unroll
        for (int j = 0; j < N; j++) {
            cd s = mk(0.0, 0.0);
#pragma unroll
            for (int k = 0; k < N; k++) s = cfma(A[i][k], B[k][j], s);
            C[i][j] = s;
        }
}
struct ExpcArgs {
    SysParams sp;
    // what the values take of the masses and charges, so that no thread
    // divides by them
    double im2[NMAX + 1], im3[NMAX + 1];  // 1 / m^2, 1 / m^3 of m0, m1..mn
    double cw[NMAX][NMAX];       // (m_k + m_p) / (m_k m_p)^2, k < p; [p][p]: with m0 for m_k
    double wq[NMAX][NMAX];       // q0 q_a, or q_a q_b for a < b
    double wdw[NMAX][NMAX];      // wq (1 / m0^2 + 1 / m_a^2), or with m_a, m_b
    double woo[NMAX][NMAX];      // wq / (m0 m_a), or -wq / (m_a m_b)
    double icm[NMAX][NMAX];      // 1 / (2 pi (M_aa or M_aa + M_bb - 2 M_ab))
    double bvc[NMAX][NMAX + 1];  // Glob_bvc
    double energy;               // Glob_CurrEnergy
    double err_mult;             // 2 (SymmAdaptMethod 1) or 3 (2)
    int nterms;
    int nv;                      // 6 np + 9
    long long npairs;
};

// Weighted accumulation of the values in MEkl order (src/workproc.f90:
// 8218-8225), four at a time: their weights and error bounds are summed over
// the warp, and lane l keeps the running sum of entry l / 4 of each group
// (entries 2k and 2k + 1: weight and bound of the group's value k).  A thread
// of the warp without a pair has w = 0.
template <int NV>
struct Acc {
    static constexpr int G = (NV + 3) / 4;
    double sum[G];
    double buf[8];
    double p1, p2;                 // Re(c_i^* c_j), -Im(c_i^* c_j)
    double rci, ici, rcj, icj;
    double w, em;
    __device__ __forceinline__ void zero()
    {
#pragma unroll
        for (int g = 0; g < G; g++) sum[g] = 0.0;
#pragma unroll
        for (int k = 0; k < 8; k++) buf[k] = 0.0;
    }
    __device__ __forceinline__ void add(int a, cd O)
    {
        const double beta = p1 * O.x + p2 * O.y;
        const double mu = fabs(rci * (rcj * O.x - icj * O.y)) + fabs(rcj * (rci * O.x + ici * O.y)) +
                          fabs(ici * (icj * O.x + rcj * O.y)) + fabs(icj * (ici * O.x - rci * O.y));
        buf[2 * (a & 3)] = w * beta;
        buf[2 * (a & 3) + 1] = fabs(w * (mu + em * fabs(beta)));
        if ((a & 3) == 3 || a == NV - 1) {
            sum[a >> 2] += warp_transpose_sum<8>(buf);
#pragma unroll
            for (int k = 0; k < 8; k++) buf[k] = 0.0;
        }
    }
};

__device__ __forceinline__ void pair_of(long long p, int& i, int& j)
{
    long long r = (long long)((sqrt(8.0 * (double)p + 1.0) - 1.0) * 0.5);
    while (r * (r + 1) / 2 > p) r--;
    while ((r + 1) * (r + 2) / 2 <= p) r++;
    i = (int)r;
    j = (int)(p - r * (r + 1) / 2);
}

// Unpacked bra / ket of one pair: L L' and B (src/matelem.f90:1038-1072).
template <int N>
__device__ __forceinline__ void unpack(const double* __restrict__ par, double (&A)[N][N], double (&B)[N][N],
                                       double& det)
{
    constexpr int NP = N * (N + 1) / 2;
    double L[N][N];
    int idx = 0;
#pragma unroll
    for (int i = 0; i < N; i++)
#pragma unroll
        for (int j = i; j < N; j++, idx++) {
            L[i][j] = 0.0;
            L[j][i] = __ldg(par + idx);
            B[i][j] = __ldg(par + NP + idx);
            B[j][i] = B[i][j];
        }
    det = 1.0;
#pragma unroll
    for (int i = 0; i < N; i++) det *= L[i][i];
#pragma unroll
    for (int i = 0; i < N; i++)
#pragma unroll
        for (int j = i; j < N; j++) {
            double s = 0.0;
#pragma unroll
            for (int k = 0; k <= j; k++) s = fma(L[i][k], L[j][k], s);
            A[i][j] = s;
            A[j][i] = s;
        }
}

// P' X P for an integer-valued matrix P (src/matelem.f90:1074-1125)
template <int N>
__device__ __forceinline__ void congruence(const double (&X)[N][N], const double* __restrict__ P, double (&R)[N][N])
{
    double W[N][N];
#pragma unroll
    for (int i = 0; i < N; i++)
#pragma unroll
        for (int j = 0; j < N; j++) {
            double s = 0.0;
#pragma unroll
            for (int k = 0; k < N; k++) s = fma(__ldg(P + k * NMAX + i), X[k][j], s);
            W[i][j] = s;
        }
#pragma unroll
    for (int i = 0; i < N; i++)
#pragma unroll
        for (int j = i; j < N; j++) {
            double s = 0.0;
#pragma unroll
            for (int k = 0; k < N; k++) s = fma(W[i][k], __ldg(P + k * NMAX + j), s);
            R[i][j] = s;
            R[j][i] = s;
        }
}

// C = tCk + tCl = L D L' (its pivots are the squares of those of the
// pseudo-Cholesky factor of src/matelem.f90:1152-1201), its inverse and the
// overlap.
template <int N>
__device__ __forceinline__ void inverse_overlap(const cd (&C)[N][N], double absdet, double two_r3n2,
                                                cd (&inv)[N][N], cd& S)
{
    cd L[N][N], G[N][N], X[N][N], r[N];
    cd det = mk(1.0, 0.0);
#pragma unroll
    for (int i = 0; i < N; i++) {
        cd d = C[i][i];
#pragma unroll
        for (int k = 0; k < i; k++) d = cfms(L[i][k], G[i][k], d);
        det = (i == 0) ? d : det * d;
        r[i] = crcp_series(d);
#pragma unroll
        for (int j = i + 1; j < N; j++) {
            cd g = C[i][j];
#pragma unroll
            for (int k = 0; k < i; k++) g = cfms(L[j][k], G[i][k], g);
            G[j][i] = g;
            L[j][i] = cmul(g, r[i]);
        }
    }
#pragma unroll
    for (int j = 1; j < N; j++)
#pragma unroll
        for (int i = j - 1; i >= 0; i--) {
            cd s = -L[j][i];
#pragma unroll
            for (int k = i + 1; k < j; k++) s = cfms(L[j][k], X[k][i], s);
            X[j][i] = s;
        }
#pragma unroll
    for (int j = 0; j < N; j++)
#pragma unroll
        for (int i = 0; i <= j; i++) {
            cd s = (i == j) ? r[j] : cmul(r[j], X[j][i]);
#pragma unroll
            for (int k = j + 1; k < N; k++) s = cfma(cmul(r[k], X[k][j]), X[k][i], s);
            inv[i][j] = s;
            inv[j][i] = s;
        }
    // c = absdet / det, S = 2^(3n/2) c sqrt(c)
    const double q = rsqrt_series(normal_range(cnorm2(det)));
    const double m = absdet * q;  // |c|
    const cd c = mk(m * q * det.x, -m * q * det.y);
    const double u = 0.5 * (fabs(c.x) + m);
    const double ri = rsqrt_series(u);
    const bool pos = c.x >= 0.0, tiny = !(u > 1e-300);  // a vanishing overlap
    const double t = u * ri, h = 0.5 * c.y * ri;
    const cd sc = tiny ? cd{0.0 * u, 0.0} : cd{pos ? t : fabs(h), pos ? h : copysign(t, c.y)};
    S = two_r3n2 * cmul(c, sc);
}

// The permuted bra tCk = tAk - i tBk and ket tCl = tAl + i tBl of one term.
template <int N>
__device__ __forceinline__ void term_matrices(const double (&Ak)[N][N], const double (&Bk)[N][N],
                                              const double (&Al)[N][N], const double (&Bl)[N][N],
                                              const double* __restrict__ Pb, const double* __restrict__ Pk,
                                              cd (&tCk)[N][N], cd (&tCl)[N][N])
{
    double R1[N][N], R2[N][N];
    congruence(Ak, Pb, R1);
    congruence(Bk, Pb, R2);
#pragma unroll
    for (int i = 0; i < N; i++)
#pragma unroll
        for (int j = 0; j < N; j++) tCk[i][j] = mk(R1[i][j], -R2[i][j]);
    congruence(Al, Pk, R1);
    congruence(Bl, Pk, R2);
#pragma unroll
    for (int i = 0; i < N; i++)
#pragma unroll
        for (int j = 0; j < N; j++) tCl[i][j] = mk(R1[i][j], R2[i][j]);
}

// arcsin(z) / z, what 1/(r_P r_Q) takes of z = u_Q' C^-1 u_P / sqrt(TrCJ_P
// TrCJ_Q) (src/matelem.f90:1302-1339), as -i log(i z + sqrt(1 - z^2)) / z;
// 1 at z = 0.  Even in z, so the sign of the reference's sqrt(TrCJCJ) does
// not matter.
__device__ __forceinline__ cd asin_ratio(cd z)
{
    const cd w = mk(fma(-z.x, z.x, fma(z.y, z.y, 1.0)), -2.0 * z.x * z.y);
    // sqrt(w) on the principal branch, Re >= 0
    const double m2 = cnorm2(w);
    const double q = rsqrt_series(normal_range(m2));
    const double m = m2 * q;
    const double u = 0.5 * (fabs(w.x) + m);
    const double ri = rsqrt_series(normal_range(u));
    const double t = u * ri, h = 0.5 * w.y * ri;
    const cd sw = w.x >= 0.0 ? mk(t, h) : mk(fabs(h), copysign(t, w.y));
    const cd l = mk(sw.x - z.y, sw.y + z.x);
    const cd a = mk(atan2(l.y, l.x), -0.5 * log(cnorm2(l)));
    const cd o = cmul(a, crcp_series(z));
    const bool zero = z.x == 0.0 && z.y == 0.0;
    return mk(zero ? 1.0 : o.x, zero ? 0.0 : o.y);
}

// 1/(r_P r_Q), P before Q in vech order, are computed EXPC_PQ at a time: the
// z go to the thread's column of shared memory, one loop takes them to
// arcsin(z) / z, and the unrolled code reads these back.  (Unrolled, the
// logarithms of all pairs are more code than the instruction cache holds;
// a loop over the pairs themselves spends its time on selecting operands.)
constexpr int EXPC_PQ = 15;
// vech pair index of (P, Q), P < Q < np, and back
__host__ __device__ constexpr int pq_count(int np) { return np * (np - 1) / 2; }

// values per pair term, and their MEkl indices: all are produced by k_expc
template <int N>
__host__ __device__ constexpr int expc_nv() { return 6 * (N * (N + 1) / 2) + 9; }

// All 6 np + 9 values of the pairs of one CTA, summed: partial[CTA][values,
// then bounds].  Bound by FP64 arithmetic at two CTAs an SM (255 registers):
// the arcsines of the pairs of pairs are most of it (15 for n = 3).  K =
// 1000, n = 3, four terms: 1.07 ms a call, with the reference's sums term by
// term in four kernels (accumulators in shared memory, divisions by masses
// and branching roots in every thread) 4.9 ms; n = 2 0.24 and 0.98 ms, n =
// 4, K = 150, 14 terms 1.0 and 2.4 ms.  Three CTAs an SM: 1.24 ms.
template <int N>
__global__ void __launch_bounds__(EXPC_BLK, EXPC_MINB)
    k_expc(const double* __restrict__ params, int npt, const cd* __restrict__ cvec, const double* __restrict__ diagS,
           const double* __restrict__ terms, const __grid_constant__ ExpcArgs ea, double* __restrict__ partial)
{
    constexpr int NP = N * (N + 1) / 2;
    constexpr int NV = expc_nv<N>();
    constexpr int NPQ = pq_count(NP);
    __shared__ double2 zsm[EXPC_PQ < NPQ ? EXPC_PQ : NPQ][EXPC_BLK];
    __shared__ double red[EXPC_BLK / 32][Acc<NV>::G * 8];
    const int tid = threadIdx.x, lane = tid & 31;
    const SysParams& sp = ea.sp;
    Acc<NV> acc;
    acc.zero();
    acc.em = ea.err_mult;
    for (long long base = (long long)blockIdx.x * EXPC_BLK; base < ea.npairs; base += (long long)gridDim.x * EXPC_BLK) {
        const bool active = base + tid < ea.npairs;
        int pi, pj;
        pair_of(active ? base + tid : 0, pi, pj);
        double Ak[N][N], Bk[N][N], Al[N][N], Bl[N][N], dk, dl;
        unpack<N>(params + (size_t)pi * npt, Ak, Bk, dk);
        unpack<N>(params + (size_t)pj * npt, Al, Bl, dl);
        const double absdet = fabs(dl * dk);
        const cd ci = cvec[pi], cj = cvec[pj];
        double factor = (pi == pj) ? 1.0 / sqrt(diagS[pi] * diagS[pi]) : 2.0 / sqrt(diagS[pi] * diagS[pj]);
        if (!active) factor = 0.0;
        acc.rci = ci.x; acc.ici = ci.y; acc.rcj = cj.x; acc.icj = cj.y;
        acc.p1 = ci.x * cj.x + ci.y * cj.y;
        acc.p2 = ci.y * cj.x - ci.x * cj.y;
        for (int t = 0; t < ea.nterms; t++) {
            const double* tp = terms + (size_t)t * (2 * NMAX * NMAX + 2);
            acc.w = factor * __ldg(tp + 2 * NMAX * NMAX) * __ldg(tp + 2 * NMAX * NMAX + 1);
            cd inv[N][N], X[N][N], Vk[N][N], Vl[N][N], S;
            {
                cd tCk[N][N], tCl[N][N], C[N][N];
                term_matrices<N>(Ak, Bk, Al, Bl, tp, tp + NMAX * NMAX, tCk, tCl);
#pragma unroll
                for (int i = 0; i < N; i++)
#pragma unroll
                    for (int j = 0; j < N; j++) C[i][j] = tCk[i][j] + tCl[i][j];
                inverse_overlap<N>(C, absdet, sp.two_r3n2, inv, S);
                mm(inv, tCk, Vk);
                mm(inv, tCl, Vl);
#pragma unroll
                for (int i = 0; i < N; i++)
#pragma unroll
                    for (int j = i; j < N; j++) {
                        cd s = mk(0.0, 0.0);
#pragma unroll
                        for (int k = 0; k < N; k++) s = cfma(tCk[i][k], Vl[k][j], s);
                        X[i][j] = s;
                        X[j][i] = s;
                    }
            }
            const cd cn = TWO_OVER_SQRTPI * S;
            const cd cdl = (1.0 / (PI_D * SQRTPI)) * S;
            // 1/sqrt(TrCJ_P) and 1/TrCJ_P
            cd tr[NP], rs[NP], rt[NP], rm[NP];
            double wq[NP];
            {
                int P = 0;
#pragma unroll
                for (int a = 0; a < N; a++)
#pragma unroll
                    for (int b = a; b < N; b++, P++) {
                        // inv(i,i) + inv(j,j) - inv(j,i) - inv(j,i), src/matelem.f90:1252
                        tr[P] = (a == b) ? inv[a][a] : inv[a][a] + inv[b][b] - inv[b][a] - inv[b][a];
                        rs[P] = crsqrt(tr[P], rt[P]);
                        rm[P] = cn * rs[P];  // <1/r_P>
                        wq[P] = ea.wq[a][b];
                    }
            }
            // 1/r^2, 1/r, r, r^2, delta(r), src/matelem.f90:1231-1268; Darwin
            // from delta(r), src/matelem.f90:1850-1873
#pragma unroll
            for (int P = 0; P < NP; P++) acc.add(P, (2.0 * S) * rt[P]);
#pragma unroll
            for (int P = 0; P < NP; P++) acc.add(NP + P, rm[P]);
#pragma unroll
            for (int P = 0; P < NP; P++) acc.add(2 * NP + P, cn * (tr[P] * rs[P]));
#pragma unroll
            for (int P = 0; P < NP; P++) acc.add(3 * NP + P, (1.5 * S) * tr[P]);
            cd dw = mk(0.0, 0.0);
            {
                int P = 0;
#pragma unroll
                for (int a = 0; a < N; a++)
#pragma unroll
                    for (int b = a; b < N; b++, P++) {
                        const cd dr = cdl * (rs[P] * rt[P]);
                        acc.add(4 * NP + P, dr);
                        dw = rfma(ea.wdw[a][b], dr, dw);
                    }
            }
            // tr[M X]; rows of X summed; 1'X1
            cd trM = mk(0.0, 0.0), sX[N], s1 = mk(0.0, 0.0);
#pragma unroll
            for (int i = 0; i < N; i++) {
                sX[i] = mk(0.0, 0.0);
#pragma unroll
                for (int k = 0; k < N; k++) {
                    trM = rfma(sp.M[i * NMAX + k], X[k][i], trM);
                    sX[i] = sX[i] + X[k][i];
                }
                s1 = s1 + sX[i];
            }
            // mass-velocity, src/matelem.f90:1487-1597
            cd mv = ea.im3[0] * (s1 * s1);
#pragma unroll
            for (int i = 0; i < N; i++)
                mv = rfma(ea.im3[i + 1], X[i][i] * X[i][i], mv);
            mv = -7.5 * (S * mv);
            // Drachmanised mass-velocity (src/matelem.f90:1675-1848) and Darwin
            // (src/matelem.f90:1875-1929): W1 = 1/m0^2 + diag(1/m_i^2)
            cd trW = ea.im2[0] * s1;
#pragma unroll
            for (int i = 0; i < N; i++) trW = rfma(ea.im2[i + 1], X[i][i], trW);
            cd dd = mk(0.0, 0.0);  // the ME_dXd_dYd terms, over S/8
#pragma unroll
            for (int p = 0; p < N; p++) {
                dd = rfma(ea.cw[p][p], 36.0 * (s1 * X[p][p]) + 24.0 * (sX[p] * sX[p]), dd);
#pragma unroll
                for (int k = 0; k < p; k++)
                    dd = rfma(ea.cw[k][p], 36.0 * (X[k][k] * X[p][p]) + 24.0 * (X[k][p] * X[k][p]), dd);
            }
            dd = 0.125 * (S * dd) - (1.5 * ea.energy) * (S * trW);
            // orbit-orbit, src/matelem.f90:1394-1485
            cd oo = mk(0.0, 0.0);
            // the sums over pairs: Drachmanised delta (src/matelem.f90:1349-1392,
            // num without its 1/(r_P r_Q)) and the second Drachmanised terms
            cd num[NP], V = mk(0.0, 0.0);
            {
                int P = 0;
#pragma unroll
                for (int a = 0; a < N; a++)
#pragma unroll
                    for (int b = a; b < N; b++, P++) {
                        V = rfma(wq[P], rm[P], V);
                        oo = rfma(ea.woo[a][b], rm[P] * (a == b ? sX[a] : X[a][b]), oo);
                        // tCk C^-1 u_P, tCl C^-1 u_P
                        cd yk[N], yl[N];
#pragma unroll
                        for (int m = 0; m < N; m++) {
                            yk[m] = a == b ? Vk[a][m] : Vk[a][m] - Vk[b][m];
                            yl[m] = a == b ? Vl[a][m] : Vl[a][m] - Vl[b][m];
                        }
                        cd tM = mk(0.0, 0.0), tW = mk(0.0, 0.0), ys = mk(0.0, 0.0);
#pragma unroll
                        for (int m = 0; m < N; m++) {
                            cd u = mk(0.0, 0.0);
#pragma unroll
                            for (int k = 0; k < N; k++) u = rfma(sp.M[m * NMAX + k], yl[k], u);
                            tM = cfma(yk[m], u, tM);
                            tW = rfma(ea.im2[m + 1], yl[m] * yl[m], tW);
                            ys = ys + yl[m];
                        }
                        tW = rfma(ea.im2[0], ys * ys, tW);
                        dd = rfma(wq[P], rm[P] * (1.5 * trW + 0.5 * (tW * rt[P])), dd);
                        num[P] = rm[P] * (mk(ea.energy, 0.0) - 6.0 * trM + 2.0 * (tM * rt[P])) -
                                 wq[P] * ((2.0 * S) * rt[P]);
                    }
            }
            // 1/(r_P r_Q), P before Q
            const cd cpq = (4.0 / PI_D) * S;
#pragma unroll
            for (int ch = 0; ch * EXPC_PQ < NPQ; ch++) {
                int e = 0, P = 0;
#pragma unroll
                for (int a = 0; a < N; a++)
#pragma unroll
                    for (int b = a; b < N; b++, P++) {
                        int Q = 0;
#pragma unroll
                        for (int c = 0; c < N; c++)
#pragma unroll
                            for (int d = c; d < N; d++, Q++) {
                                if (Q <= P) continue;
                                if (e / EXPC_PQ == ch) {
                                    cd x = mk(0.0, 0.0);
                                    if (!(a == b && a < c && c < d)) {  // (see the file header)
                                        x = a == b ? inv[a][c] : inv[a][c] - inv[b][c];
                                        if (c != d) x = x - (a == b ? inv[a][d] : inv[a][d] - inv[b][d]);
                                    }
                                    x = x * (rs[P] * rs[Q]);
                                    zsm[e % EXPC_PQ][tid] = make_double2(x.x, x.y);
                                }
                                e++;
                            }
                    }
#pragma unroll 1
                for (int k = 0; k < (NPQ - ch * EXPC_PQ < EXPC_PQ ? NPQ - ch * EXPC_PQ : EXPC_PQ); k++) {
                    const double2 z = zsm[k][tid];
                    const cd r = asin_ratio(mk(z.x, z.y));
                    zsm[k][tid] = make_double2(r.x, r.y);
                }
                e = 0;
#pragma unroll
                for (int P2 = 0; P2 < NP; P2++)
#pragma unroll
                    for (int Q = P2 + 1; Q < NP; Q++, e++)
                        if (e / EXPC_PQ == ch) {
                            const double2 z = zsm[e % EXPC_PQ][tid];
                            const cd R = (cpq * (rs[P2] * rs[Q])) * mk(z.x, z.y);
                            num[P2] = rfma(-wq[Q], R, num[P2]);
                            num[Q] = rfma(-wq[P2], R, num[Q]);
                        }
            }
            {
                int P = 0;
#pragma unroll
                for (int a = 0; a < N; a++)
#pragma unroll
                    for (int b = a; b < N; b++, P++) {
                        acc.add(5 * NP + P, ea.icm[a][b] * num[P]);
                    }
            }
            const cd T = 6.0 * (S * trM);  // src/matelem.f90:1203-1229
            acc.add(6 * NP + 0, T + V);
            acc.add(6 * NP + 1, S);
            acc.add(6 * NP + 2, T);
            acc.add(6 * NP + 3, V);
            acc.add(6 * NP + 4, mv);
            acc.add(6 * NP + 5, dd);
            acc.add(6 * NP + 6, (-0.5 * PI_D) * dw);
            acc.add(6 * NP + 7, dd);
            acc.add(6 * NP + 8, 4.0 * oo);
        }
    }
    if ((lane & 3) == 0)
#pragma unroll
        for (int g = 0; g < Acc<NV>::G; g++) red[tid >> 5][g * 8 + (lane >> 2)] = acc.sum[g];
    __syncthreads();
    for (int l = tid; l < 2 * NV; l += EXPC_BLK) {
        double s = 0.0;
        for (int wp = 0; wp < EXPC_BLK / 32; wp++) s += red[wp][l];
        partial[(size_t)blockIdx.x * 2 * NV + (l & 1) * NV + (l >> 1)] = s;
    }
}

// Correlation functions (np per grid point) and particle densities (n+1
// per grid point), src/matelem.f90:1931-1960; blockIdx.y selects a chunk
// of `gchunk` grid entries (grid points times values).
template <int N>
__global__ void __launch_bounds__(GRID_BLK) k_expc_grid(const double* __restrict__ params, int npt,
                                                        const cd* __restrict__ cvec, const double* __restrict__ diagS,
                                                        const double* __restrict__ terms, ExpcArgs ea,
                                                        const double* __restrict__ cf_grid, int ncf,
                                                        const double* __restrict__ dens_grid, int ndens, int gchunk,
                                                        double* __restrict__ partial, int ngrid)
{
    constexpr int NP = N * (N + 1) / 2;
    extern __shared__ double sacc[];
    const int tid = threadIdx.x;
    const int g0 = blockIdx.y * gchunk;
    const int g1 = min(ngrid, g0 + gchunk);
    for (int g = g0; g < g1; g++) sacc[(g - g0) * GRID_BLK + tid] = 0.0;
    const SysParams& sp = ea.sp;
    for (long long pidx = (long long)blockIdx.x * GRID_BLK + tid; pidx < ea.npairs;
         pidx += (long long)gridDim.x * GRID_BLK) {
        int pi, pj;
        pair_of(pidx, pi, pj);
        double Ak[N][N], Bk[N][N], Al[N][N], Bl[N][N], dk, dl;
        unpack<N>(params + (size_t)pi * npt, Ak, Bk, dk);
        unpack<N>(params + (size_t)pj * npt, Al, Bl, dl);
        const double absdet = fabs(dl * dk);
        const cd ci = cvec[pi], cj = cvec[pj];
        const double factor = (pi == pj) ? 1.0 / sqrt(diagS[pi] * diagS[pi]) : 2.0 / sqrt(diagS[pi] * diagS[pj]);
        const double p1 = ci.x * cj.x + ci.y * cj.y, p2 = ci.y * cj.x - ci.x * cj.y;
        for (int t = 0; t < ea.nterms; t++) {
            const double* tp = terms + (size_t)t * (2 * NMAX * NMAX + 2);
            const double w = factor * __ldg(tp + 2 * NMAX * NMAX) * __ldg(tp + 2 * NMAX * NMAX + 1);
            cd tCk[N][N], tCl[N][N], inv[N][N], S;
            term_matrices<N>(Ak, Bk, Al, Bl, tp, tp + NMAX * NMAX, tCk, tCl);
#pragma unroll
            for (int i = 0; i < N; i++)
#pragma unroll
                for (int j = 0; j < N; j++) tCk[i][j] = tCk[i][j] + tCl[i][j];
            inverse_overlap<N>(tCk, absdet, sp.two_r3n2, inv, S);
            const cd pre = (1.0 / (PI_D * SQRTPI)) * S;
            // TrCJ in vech order, then the density quadratic forms
            cd x[NP + N + 1];
            {
                int P = 0;
#pragma unroll
                for (int a = 0; a < N; a++)
#pragma unroll
                    for (int b = a; b < N; b++, P++)
                        x[P] = (a == b) ? inv[a][a] : inv[a][a] + inv[b][b] - inv[b][a] - inv[b][a];
            }
#pragma unroll
            for (int i = 0; i <= N; i++) {
                cd s = mk(0.0, 0.0);
#pragma unroll
                for (int p = 0; p < N; p++) {
                    s = rfma(ea.bvc[p][i] * ea.bvc[p][i], inv[p][p], s);
#pragma unroll
                    for (int q = p + 1; q < N; q++) s = rfma(2.0 * ea.bvc[q][i] * ea.bvc[p][i], inv[q][p], s);
                }
                x[NP + i] = s;
            }
            cd xr[NP + N + 1], px[NP + N + 1];  // 1/x and pre/(sqrt(x) x)
#pragma unroll
            for (int v = 0; v < NP + N + 1; v++) {
                const cd rs = crsqrt(x[v], xr[v]);
                px[v] = pre * (rs * xr[v]);
            }
            for (int g = g0; g < g1; g++) {
                int v, k;
                double r;
                if (g < ncf * NP) {
                    k = g / NP;
                    v = g - k * NP;
                    r = cf_grid[k];
                } else {
                    const int gd = g - ncf * NP;
                    k = gd / (N + 1);
                    v = NP + (gd - k * (N + 1));
                    r = dens_grid[k];
                }
                cd O = mk(0.0, 0.0);
#pragma unroll
                for (int u = 0; u < NP + N + 1; u++)
                    if (u == v) O = px[u] * cexp_((-r * r) * xr[u]);
                sacc[(g - g0) * GRID_BLK + tid] += w * (p1 * O.x + p2 * O.y);
            }
        }
    }
    __syncthreads();
    for (int g = g0 + tid; g < g1; g += GRID_BLK) {
        double s = 0.0;
        for (int t = 0; t < GRID_BLK; t++) s += sacc[(g - g0) * GRID_BLK + t];
        partial[(size_t)blockIdx.x * ngrid + g] = s;
    }
}

// out[a] = sum over blocks of partial[b][a], one CTA a value, in a fixed
// order; the second half (the error bounds) times epsilon when `eps_from` <
// count.
__global__ void __launch_bounds__(128) k_expc_sum(const double* __restrict__ partial, int nblocks, int count,
                                                  int eps_from, double* __restrict__ out)
{
    __shared__ double sh[128];
    const int a = blockIdx.x;
    double s = 0.0;
    for (int b = threadIdx.x; b < nblocks; b += 128) s += partial[(size_t)b * count + a];
    sh[threadIdx.x] = s;
    for (int h = 64; h >= 1; h >>= 1) {
        __syncthreads();
        if (threadIdx.x < h) sh[threadIdx.x] += sh[threadIdx.x + h];
    }
    if (threadIdx.x == 0) out[a] = (a >= eps_from) ? sh[0] * DBL_EPSILON : sh[0];
}

template <int N>
int launch_n(Ctx& c, const ExpcArgs& ea, const double* terms, const cd* cvec, const double* cfg, int ncf,
             const double* dg, int ndens, double* partial, int nblocks, double* out, double* gpartial, int gblocks,
             int gchunk, int ngrid, double* gout)
{
    k_expc<N><<<nblocks, EXPC_BLK, 0, c.stream>>>(c.params, c.npt, cvec, c.diagS, terms, ea, partial);
    k_expc_sum<<<2 * ea.nv, 128, 0, c.stream>>>(partial, nblocks, 2 * ea.nv, ea.nv, out);
    c.launches += 2;
    if (ngrid > 0) {
        const size_t gsm = (size_t)gchunk * GRID_BLK * sizeof(double);
        if (cudaFuncSetAttribute(k_expc_grid<N>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)gsm) !=
            cudaSuccess)
            return -2;
        dim3 grid(gblocks, (ngrid + gchunk - 1) / gchunk);
        k_expc_grid<N><<<grid, GRID_BLK, gsm, c.stream>>>(c.params, c.npt, cvec, c.diagS, terms, ea, cfg, ncf, dg,
                                                          ndens, gchunk, gpartial, ngrid);
        k_expc_sum<<<ngrid, 128, 0, c.stream>>>(gpartial, gblocks, ngrid, ngrid, gout);
        c.launches += 2;
    }
    return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

}  // namespace

int expectation_values(Ctx& c, int nbasis, const double* masses, int nterms, const int* pbra, const int* pket,
                       const double* coef1, const double* coef2, int err_mult, double energy, const cd* c_host,
                       int ncf, const double* cf_grid, int ndens, const double* dens_grid, double* values,
                       double* errors, double* cf, double* dens)
{
    const int n = c.n, np = c.np;
    if (nbasis < 1 || nbasis > c.ld || nterms < 1 || ncf < 0 || ndens < 0) return -1;
    ExpcArgs ea{};
    ea.sp = c.sp;
    double mtot = 0.0;
    for (int i = 0; i <= n; i++) {
        const double m = masses[i];
        mtot += m;
        ea.im2[i] = 1.0 / (m * m);
        ea.im3[i] = 1.0 / (m * m * m);
    }
    for (int a = 0; a < n; a++)
        for (int b = a; b < n; b++) {
            // a = b: the pair of particle a with particle 0
            const double ma = a == b ? masses[0] : masses[a + 1], mb = masses[b + 1];
            const double(&M)[NMAX * NMAX] = c.sp.M;
            ea.wq[a][b] = a == b ? c.sp.q0 * c.sp.q[a] : c.sp.q[a] * c.sp.q[b];
            ea.cw[a][b] = (ma + mb) / (ma * ma * mb * mb);
            ea.wdw[a][b] = (1.0 / (ma * ma) + 1.0 / (mb * mb)) * ea.wq[a][b];
            ea.woo[a][b] = (a == b ? 1.0 : -1.0) * ea.wq[a][b] / (ma * mb);
            ea.icm[a][b] = 1.0 / (2.0 * PI_D *
                                  (a == b ? M[a * NMAX + a]
                                          : M[a * NMAX + a] + M[b * NMAX + b] - M[a * NMAX + b] - M[a * NMAX + b]));
        }
    // Glob_bvc, src/workproc.f90:612-621
    for (int i = 0; i <= n; i++)
        for (int p = 0; p < n; p++) ea.bvc[p][i] = -masses[p + 1] / mtot;
    for (int i = 1; i <= n; i++) ea.bvc[i - 1][i] += 1.0;
    ea.energy = energy;
    ea.err_mult = err_mult;
    ea.nterms = nterms;
    ea.nv = 6 * np + 9;
    ea.npairs = (long long)nbasis * (nbasis + 1) / 2;

    // term list: Pbra, Pket (row-major NMAX x NMAX doubles), coef1, coef2
    const int tstride = 2 * NMAX * NMAX + 2;
    std::vector<double> th((size_t)nterms * tstride, 0.0);
    for (int t = 0; t < nterms; t++) {
        double* d = th.data() + (size_t)t * tstride;
        for (int i = 0; i < n; i++)
            for (int j = 0; j < n; j++) {
                d[i * NMAX + j] = pbra[(size_t)t * n * n + i + j * n];
                d[NMAX * NMAX + i * NMAX + j] = pket[(size_t)t * n * n + i + j * n];
            }
        d[2 * NMAX * NMAX] = coef1[t];
        d[2 * NMAX * NMAX + 1] = coef2 ? coef2[t] : 1.0;
    }
    int sms = 148;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, c.dev);
    const long long blocks_needed = (ea.npairs + EXPC_BLK - 1) / EXPC_BLK;
    const int nblocks = (int)std::min<long long>(blocks_needed, (long long)sms * EXPC_MINB * 2);
    const int ngrid = ncf * np + ndens * (n + 1);
    const int gchunk = 48;  // 48 x 64 doubles of shared memory per block
    const int gblocks = (int)std::min<long long>((ea.npairs + GRID_BLK - 1) / GRID_BLK, (long long)sms * 2);

    double *d_terms = nullptr, *d_part = nullptr, *d_out = nullptr, *d_gpart = nullptr, *d_gout = nullptr,
           *d_cfg = nullptr, *d_dg = nullptr;
    cd* d_c = nullptr;
    int rc = 0;
    auto alloc = [&](void** p, size_t bytes) {
        if (bytes == 0) return true;
        if (cudaMalloc(p, bytes) != cudaSuccess) {
            cudaGetLastError();
            rc = -3;
            return false;
        }
        return true;
    };
    const size_t nv = ea.nv;
    if (alloc((void**)&d_terms, th.size() * sizeof(double)) &&
        alloc((void**)&d_part, (size_t)nblocks * 2 * nv * sizeof(double)) &&
        alloc((void**)&d_out, 2 * nv * sizeof(double)) &&
        alloc((void**)&d_gpart, (size_t)gblocks * ngrid * sizeof(double)) &&
        alloc((void**)&d_gout, (size_t)ngrid * sizeof(double)) &&
        alloc((void**)&d_cfg, (size_t)ncf * sizeof(double)) && alloc((void**)&d_dg, (size_t)ndens * sizeof(double)) &&
        (c_host == nullptr || alloc((void**)&d_c, (size_t)nbasis * sizeof(cd)))) {
        cudaStream_t s = c.stream;
        bool ok = cudaMemcpyAsync(d_terms, th.data(), th.size() * sizeof(double), cudaMemcpyHostToDevice, s) ==
                  cudaSuccess;
        if (ncf) ok = ok && cudaMemcpyAsync(d_cfg, cf_grid, ncf * sizeof(double), cudaMemcpyHostToDevice, s) ==
                                cudaSuccess;
        if (ndens)
            ok = ok && cudaMemcpyAsync(d_dg, dens_grid, ndens * sizeof(double), cudaMemcpyHostToDevice, s) ==
                           cudaSuccess;
        if (c_host) ok = ok && cudaMemcpyAsync(d_c, c_host, nbasis * sizeof(cd), cudaMemcpyHostToDevice, s) ==
                                   cudaSuccess;
        c.bytes_h2d += th.size() * sizeof(double) + (ncf + ndens) * sizeof(double) +
                       (c_host ? nbasis * sizeof(cd) : 0);
        const cd* cv = c_host ? d_c : c.c;
        if (!ok) rc = -2;
        if (rc == 0) {
            switch (n) {
                case 2: rc = launch_n<2>(c, ea, d_terms, cv, d_cfg, ncf, d_dg, ndens, d_part, nblocks, d_out, d_gpart,
                                         gblocks, gchunk, ngrid, d_gout); break;
                case 3: rc = launch_n<3>(c, ea, d_terms, cv, d_cfg, ncf, d_dg, ndens, d_part, nblocks, d_out, d_gpart,
                                         gblocks, gchunk, ngrid, d_gout); break;
                case 4: rc = launch_n<4>(c, ea, d_terms, cv, d_cfg, ncf, d_dg, ndens, d_part, nblocks, d_out, d_gpart,
                                         gblocks, gchunk, ngrid, d_gout); break;
                case 5: rc = launch_n<5>(c, ea, d_terms, cv, d_cfg, ncf, d_dg, ndens, d_part, nblocks, d_out, d_gpart,
                                         gblocks, gchunk, ngrid, d_gout); break;
                default: rc = -1;
            }
        }
        if (rc == 0) {
            std::vector<double> h(2 * nv), hg(ngrid);
            ok = cudaMemcpyAsync(h.data(), d_out, 2 * nv * sizeof(double), cudaMemcpyDeviceToHost, s) == cudaSuccess;
            if (ngrid)
                ok = ok && cudaMemcpyAsync(hg.data(), d_gout, ngrid * sizeof(double), cudaMemcpyDeviceToHost, s) ==
                               cudaSuccess;
            ok = ok && cudaStreamSynchronize(s) == cudaSuccess;
            c.bytes_d2h += (2 * nv + ngrid) * sizeof(double);
            if (!ok) {
                rc = -2;
            } else {
                for (size_t a = 0; a < nv; a++) {
                    if (values) values[a] = h[a];
                    if (errors) errors[a] = h[nv + a];
                }
                if (cf)
                    for (int g = 0; g < ncf * np; g++) cf[g] = hg[g];
                if (dens)
                    for (int g = 0; g < ndens * (n + 1); g++) dens[g] = hg[ncf * np + g];
            }
        }
        if (rc != 0) cudaStreamSynchronize(s);
    }
    cudaFree(d_terms);
    cudaFree(d_part);
    cudaFree(d_out);
    cudaFree(d_gpart);
    cudaFree(d_gout);
    cudaFree(d_cfg);
    cudaFree(d_dg);
    cudaFree(d_c);
    cudaGetLastError();
    return rc;
}

}  // namespace ecg
