// ecg_grad.cuh -- derivatives of one ECG pair term.
//
// With the eigenvalue E fixed, the derivatives of one term
// (src/matelem.f90:306-748) are
//       dH/dvechL - E dS/dvechL  (entry (j,i), j >= i)
//            = a * delta_ij / L_ii - 2 (Z L)_ji
//       dH/dvechB - E dS/dvechB  (entry (i,j), weight 1 on the diagonal,
//                                 2 off it)
//            = +i Z_ij (bra)   or   -i Z_ij (ket),
//   with a = (3/2)(H - E S) and one complex symmetric matrix Z per side:
//       Z_k = a C^-1 - C^-1 [6 S tCl M tCl + S/sqrt(pi) Q] C^-1
//       Z_l = P ( a C^-1 - C^-1 [6 S Ck M Ck + S/sqrt(pi) Q] C^-1 ) P'
//   where Q(i,i) = w_ii + sum_{j!=i} w_ij, Q(i,j) = -w_ij collects the
//   Coulomb weights w_ij = cnumb of src/matelem.f90:677-681.  This follows
//   from the reference's formulas: every Coulomb matrix tQ of
//   src/matelem.f90:609-631 is the rank-one C^-1 (e_i-e_j)(e_i-e_j)' C^-1,
//   so their weighted sum is C^-1 Q C^-1; and dS, dT, dV share the factors
//   C^-1, F = C^-1 tCl M tCl C^-1 and G = P C^-1 Ck M Ck C^-1 P'.  E = 0
//   gives dH alone, and dS has a = (3/2) S, Z = (3/2) S C^-1.
//
// Everything is S times a matrix that does not contain S, and with the unit
// lower factor of pair_term (C^-1 = X^T D^-1 X)
//       Z / S = X^T ( a' D^-1 - D^-1 (X R X^T) D^-1 ) X,
//       a' = (3/2)(h - E),  R = N6 + Qs,
// so one side costs two congruences with a unit triangular matrix (12
// complex multiply-adds each at n = 3, against 45 for inv R inv).
#pragma once
#include "ecg_math.cuh"

namespace ecg {

// r_i r_j, packed, shared by the two sides of a term.
template <int N>
__device__ __forceinline__ void pivot_products(const cd (&r)[N], cd (&rr)[Sym<N>::NP])
{
#pragma unroll
    for (int i = 0; i < N; i++)
#pragma unroll
        for (int j = i; j < N; j++) rr[vech_index(N, i, j)] = cmul(r[i], r[j]);
}

// Z (packed, vech order) = X^T (a D^-1 - D^-1 X R X^T D^-1) X for packed
// symmetric R, unit lower X (strict part read) and ar_i = a r_i.
template <int N>
__device__ __forceinline__ void adj_congruence(const cd (&X)[N][N], const cd (&rr)[Sym<N>::NP], const cd (&ar)[N],
                                               const cd (&R)[Sym<N>::NP], cd (&Z)[Sym<N>::NP])
{
    auto ix = [](int i, int j) { return i <= j ? vech_index(N, i, j) : vech_index(N, j, i); };
    // A = X R, entries (i, b <= i); then B = A X^T, lower, scaled in place
    cd A[N][N];
#pragma unroll
    for (int i = 0; i < N; i++)
#pragma unroll
        for (int b = 0; b <= i; b++) {
            cd s = R[ix(i, b)];
#pragma unroll
            for (int k = 0; k < i; k++) s = cfma(X[i][k], R[ix(k, b)], s);
            A[i][b] = s;
        }
    cd Ee[Sym<N>::NP];
#pragma unroll
    for (int i = 0; i < N; i++)
#pragma unroll
        for (int j = 0; j <= i; j++) {
            cd s = A[i][j];
#pragma unroll
            for (int b = 0; b < j; b++) s = cfma(A[i][b], X[j][b], s);
            Ee[ix(i, j)] = (i == j) ? cfms(rr[ix(i, i)], s, ar[i]) : cfms(rr[ix(i, j)], s, mk(0.0, 0.0));
        }
    // G = E X, entries (a >= j, j); then Z = X^T G, lower
#pragma unroll
    for (int a = 0; a < N; a++)
#pragma unroll
        for (int j = 0; j <= a; j++) {
            cd s = Ee[ix(a, j)];
#pragma unroll
            for (int b = j + 1; b < N; b++) s = cfma(Ee[ix(a, b)], X[b][j], s);
            A[a][j] = s;
        }
#pragma unroll
    for (int i = 0; i < N; i++)
#pragma unroll
        for (int j = 0; j <= i; j++) {
            cd s = A[i][j];
#pragma unroll
            for (int a = i + 1; a < N; a++) s = cfma(X[a][i], A[a][j], s);
            Z[ix(i, j)] = s;
        }
}

// ---------------------------------------------------------------------------
// Z <- P Z P' for the ket side.  A product of particle transpositions acts
// on the relative coordinates as rows e_x - e_b (x != b) and -e_b (the
// image of the reference particle), b one coordinate or none, in some order
// (src/workproc.f90:673-698).  perm_code packs that: b + 1 in bits 0..3
// (0: none), and for every row i the slot it is swapped with, in bits
// 4 + 3i.., so that P Z P' is a few additions and register swaps instead of
// two products with P (45 real x complex multiply-adds at n = 3).  Any other
// matrix has the code -1 and takes the general product.
// ---------------------------------------------------------------------------
__host__ __device__ inline int perm_code(const double* P, int pitch, int n)
{
    int row_slot[NMAX], b = -1;
    // b: the coordinate whose -1 stands in every row
    for (int j = 0; j < n && b < 0; j++) {
        bool all = true;
        for (int i = 0; i < n; i++) all = all && P[i * pitch + j] == -1.0;
        if (all) b = j;
    }
    bool used[NMAX] = {false, false, false, false, false};
    for (int i = 0; i < n; i++) {
        int slot = -1;
        for (int j = 0; j < n; j++) {
            const double v = P[i * pitch + j];
            if (j == b || v == 0.0) continue;
            if (v != 1.0 || slot >= 0) return -1;
            slot = j;
        }
        if (slot < 0) slot = b;  // the row -e_b
        if (slot < 0 || used[slot]) return -1;
        used[slot] = true;
        row_slot[i] = slot;
    }
    int code = b + 1, cur[NMAX];
    for (int i = 0; i < n; i++) cur[i] = i;
    for (int i = 0; i + 1 < n; i++) {
        int m = i;
        while (cur[m] != row_slot[i]) m++;
        const int c = cur[i];
        cur[i] = cur[m];
        cur[m] = c;
        code |= m << (4 + 3 * i);
    }
    return code;
}

template <int N>
__device__ __forceinline__ void perm_congruence(int code, const double* __restrict__ P, cd (&Z)[Sym<N>::NP])
{
    auto ix = [](int i, int j) { return i <= j ? vech_index(N, i, j) : vech_index(N, j, i); };
    if (code >= 0) {
        const int b = (code & 15) - 1;
        if (b >= 0) {
#pragma unroll
            for (int x = 0; x < N; x++)
                if (b == x) {
                    cd e[N];
#pragma unroll
                    for (int a = 0; a < N; a++)
                        if (a != x) e[a] = Z[ix(x, x)] - Z[ix(a, x)];
#pragma unroll
                    for (int a = 0; a < N; a++)
#pragma unroll
                        for (int c = a; c < N; c++)
                            if (a != x && c != x) Z[ix(a, c)] = (Z[ix(a, c)] - Z[ix(c, x)]) + e[a];
#pragma unroll
                    for (int a = 0; a < N; a++)
                        if (a != x) Z[ix(a, x)] = e[a];
                }
        }
#pragma unroll
        for (int i = 0; i + 1 < N; i++) {
            const int m = (code >> (4 + 3 * i)) & 7;
#pragma unroll
            for (int x = i + 1; x < N; x++)
                if (m == x) {
#pragma unroll
                    for (int a = 0; a < N; a++) {
                        if (a == i || a == x) continue;
                        const cd s = Z[ix(a, i)];
                        Z[ix(a, i)] = Z[ix(a, x)];
                        Z[ix(a, x)] = s;
                    }
                    const cd s = Z[ix(i, i)];
                    Z[ix(i, i)] = Z[ix(x, x)];
                    Z[ix(x, x)] = s;
                }
        }
        return;
    }
    cd W[N][N];
#pragma unroll
    for (int i = 0; i < N; i++)
#pragma unroll
        for (int j = 0; j < N; j++) {
            cd s = mk(0.0, 0.0);
#pragma unroll
            for (int k = 0; k < N; k++) s = rfma(__ldg(P + i * NMAX + k), Z[ix(k, j)], s);
            W[i][j] = s;
        }
#pragma unroll
    for (int i = 0; i < N; i++)
#pragma unroll
        for (int j = i; j < N; j++) {
            cd s = mk(0.0, 0.0);
#pragma unroll
            for (int k = 0; k < N; k++) s = rfma(__ldg(P + j * NMAX + k), W[i][k], s);
            Z[ix(i, j)] = s;
        }
}

// Bra and ket sides of one term over S (see the header): Zk, Zl (Zl only
// with KET, already P Zl P') and a = (3/2)(h - E).  n6l(i, j) = 6 (tCl M
// tCl)_ij.
template <int N, bool KET, typename BRA, typename KETN>
__device__ __forceinline__ cd term_adjoint(const BRA& bra, const KETN& n6l, const PairTerm<N>& te, double E,
                                           int code, const double* __restrict__ P, cd (&Zk)[Sym<N>::NP],
                                           cd (&Zl)[Sym<N>::NP])
{
    constexpr int NP = Sym<N>::NP;
    const cd a = cd{1.5 * (te.h.x - E), 1.5 * te.h.y};
    cd ar[N], rr[NP], R[NP];
#pragma unroll
    for (int i = 0; i < N; i++) ar[i] = cmul(a, te.r[i]);
    pivot_products<N>(te.r, rr);
#pragma unroll
    for (int i = 0; i < N; i++)
#pragma unroll
        for (int j = i; j < N; j++) {
            const int x = vech_index(N, i, j);
            R[x] = te.Qs[x] + n6l(i, j);
        }
    adj_congruence<N>(te.X, rr, ar, R, Zk);
    if (KET) {
#pragma unroll
        for (int i = 0; i < N; i++)
#pragma unroll
            for (int j = i; j < N; j++) {
                const int x = vech_index(N, i, j);
                R[x] = te.Qs[x] + bra.N6(i, j);
            }
        adj_congruence<N>(te.X, rr, ar, R, Zl);
        perm_congruence<N>(code, P, Zl);
    }
    return a;
}

// The derivative vector of one function (the reference's order: H-L, H-B,
// S-L, S-B blocks of NP entries) from its term sums: ZH, aH of H (E = 0),
// ZS, aS of S; isign +1 for a bra, -1 for a ket.  L lower triangular.
template <int N, typename GetH, typename GetS, typename Put>
__device__ __forceinline__ void deriv_entries(const double (&L)[N][N], const GetH& ZH, cd aH, const GetS& ZS, cd aS,
                                              double isign, const Put& put)
{
    constexpr int NP = Sym<N>::NP;
    auto half = [&](const auto& Z, cd a, int off) {
#pragma unroll
        for (int i = 0; i < N; i++)
#pragma unroll
            for (int j = i; j < N; j++) {
                cd s = mk(0.0, 0.0);
#pragma unroll
                for (int m = i; m < N; m++)
                    s = rfma(L[m][i], Z(j >= m ? vech_index(N, m, j) : vech_index(N, j, m)), s);
                cd g = -2.0 * s;
                if (i == j) g = g + (1.0 / L[i][i]) * a;
                put(off + vech_index(N, i, j), g);
                const cd z = (i == j ? isign : 2.0 * isign) * Z(vech_index(N, i, j));
                put(off + NP + vech_index(N, i, j), mk(-z.y, z.x));
            }
    };
    half(ZH, aH, 0);
    half(ZS, aS, 2 * NP);
}

}  // namespace ecg
