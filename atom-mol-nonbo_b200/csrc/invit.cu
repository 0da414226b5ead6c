// invit.cu -- one inverse-iteration step and the Rayleigh quotient of
// GHEPIIS (src/linalg.f90:1781-1926):
//   w = B^H v                  MHMV, ZGEMV('C')         (src/linalg.f90:1019-1107)
//   x = (L D L^H)^-1 w         LDLHS, 2 x ZTRSV + D^-1  (src/linalg.f90:618-775)
//   x /= max|Re x|,|Im x|      CMaxAbsReOrIm + CVScale
//   tc = x^H v / v^H v, NormOfDiff = sqrt(2n) ||x - tc v||
//   t1 = x^H B x, t2 = x^H M x VMMHMV on the lower triangles
//
// The triangular solves walk the panels of the LDL^H factor, one cooperative
// launch each with a CTA per panel (below); beyond the co-resident CTAs each
// panel step is one launch whose CTAs share the dot products against the
// already solved part, and the last CTA to finish (atomic ticket, no waiting)
// sums the partials in a fixed order and applies the panel's precomputed
// inverse block.  Results are deterministic run to run.  The host enqueues
// several steps (one where a step is a launch per panel) and the Rayleigh
// quotient at a time (ghepiis_core); launches after convergence return at
// once.
#include <algorithm>
#include <float.h>
#include "ecg_internal.h"
#include "wait_value.cuh"
#include "warp_sums.cuh"
#include "zmma.cuh"

namespace ecg {

constexpr int SOLVE_G_MAX = 64;

__device__ __forceinline__ cd ld2(const cd* p)
{
    const double2 v = __ldg(reinterpret_cast<const double2*>(p));
    return cd{v.x, v.y};
}
__device__ __forceinline__ cd ldcg2(const cd* p)
{
    const double2 v = __ldcg(reinterpret_cast<const double2*>(p));
    return cd{v.x, v.y};
}
__device__ __forceinline__ cd warp_sum(cd s)
{
#pragma unroll
    for (int o = 16; o >= 1; o >>= 1) {
        s.x += __shfl_xor_sync(0xffffffffu, s.x, o);
        s.y += __shfl_xor_sync(0xffffffffu, s.y, o);
    }
    return s;
}

// Whether a launch of the iteration has nothing to do: the host enqueues
// several iterations and the Rayleigh quotient without looking in between.
__device__ __forceinline__ bool idle(const double* red, const int* status)
{
    return red[RD_DONE] != 0.0 || status[ST_ZERO_PIVOT] != 0 || status[ST_SOLVE_TIMEOUT] != 0;
}
// The same for the Rayleigh quotient behind them.
__device__ __forceinline__ bool idle_rayleigh(const double* red, const int* status, int always)
{
    return (!always && red[RD_DONE] == 0.0) || status[ST_ZERO_PIVOT] != 0 || status[ST_SOLVE_TIMEOUT] != 0;
}

// w(i) = sum_j conj(B(j,i)) v(j); one warp per column, four accumulators.
// The solves' vectors y and x are marked as not computed on the way.
__global__ void __launch_bounds__(256) k_hemv(const cd* __restrict__ B, int ld, int n, const cd* __restrict__ v,
                                              cd* __restrict__ w, cd* __restrict__ y, cd* __restrict__ x,
                                              const double* __restrict__ red, const int* __restrict__ status)
{
    if (idle(red, status)) return;
    const int col = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (col >= n) return;
    const cd* b = B + (size_t)col * ld;
    cd s0 = mk(0.0, 0.0), s1 = s0, s2 = s0, s3 = s0;
    int j = lane;
    for (; j + 96 < n; j += 128) {
        const cd b0 = ld2(b + j), b1 = ld2(b + j + 32), b2 = ld2(b + j + 64), b3 = ld2(b + j + 96);
        s0 = cfma(conj(b0), ld2(v + j), s0);
        s1 = cfma(conj(b1), ld2(v + j + 32), s1);
        s2 = cfma(conj(b2), ld2(v + j + 64), s2);
        s3 = cfma(conj(b3), ld2(v + j + 96), s3);
    }
    for (; j < n; j += 32) s0 = cfma(conj(ld2(b + j)), ld2(v + j), s0);
    const cd s = warp_sum((s0 + s1) + (s2 + s3));
    if (lane == 0) {
        w[col] = s;
        y[col] = unset();
        x[col] = unset();
    }
}

// Forward solve of panel [j0, j1): y = Linv (w - U(0:j0, p)^H y(0:j0)),
// z = invD y.  CTA g covers rows [g*chunk, ...) of the solved part.
__global__ void __launch_bounds__(256) k_fwd(const cd* __restrict__ A, int ld, int j0, int j1, int chunk,
                                             const cd* __restrict__ w, cd* __restrict__ y, cd* __restrict__ z,
                                             const cd* __restrict__ invD, const cd* __restrict__ linv,
                                             cd* __restrict__ part, int* __restrict__ counter,
                                             const double* __restrict__ red, const int* __restrict__ status)
{
    if (idle(red, status)) return;
    __shared__ cd t[LDL_NB];
    __shared__ int last;
    const int b = j1 - j0;
    const int g = blockIdx.x, G = gridDim.x;
    const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5;
    const int i0 = g * chunk, i1 = min(j0, i0 + chunk);
    for (int m = wp; m < b; m += 8) {
        const cd* col = A + (size_t)(j0 + m) * ld;
        cd s = mk(0.0, 0.0);
        for (int i = i0 + lane; i < i1; i += 32) s = cfma(conj(ld2(col + i)), ldcg2(y + i), s);
        s = warp_sum(s);
        if (lane == 0) part[g * LDL_NB + m] = s;
    }
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) last = (atomicAdd(counter, 1) == G - 1);
    __syncthreads();
    if (!last) return;
    __threadfence();
    if (threadIdx.x < b) {
        cd s = mk(0.0, 0.0);
        for (int q = 0; q < G; q++) s = s + ldcg2(part + q * LDL_NB + threadIdx.x);
        t[threadIdx.x] = ld2(w + j0 + threadIdx.x) - s;
    }
    __syncthreads();
    if (threadIdx.x < b) {
        const int r = threadIdx.x;
        const cd* Lr = linv + (size_t)(j0 + r) * LDL_NB;
        cd s = mk(0.0, 0.0);
        for (int q = 0; q <= r; q++) s = cfma(ld2(Lr + q), t[q], s);
        y[j0 + r] = s;
        z[j0 + r] = cmul(s, ld2(invD + j0 + r));
    }
    if (threadIdx.x == 0) *counter = 0;
}

// Backward solve of panel [j0, j1): x = Linv^H (z - U(p, j1:n) x(j1:n)).
// CTA g covers columns [j1 + g*chunk, ...); 4 groups of 64 threads.
__global__ void __launch_bounds__(256) k_bwd(const cd* __restrict__ A, int ld, int j0, int j1, int n, int chunk,
                                             const cd* __restrict__ z, cd* __restrict__ x,
                                             const cd* __restrict__ linv, cd* __restrict__ part,
                                             int* __restrict__ counter, const double* __restrict__ red,
                                             const int* __restrict__ status)
{
    if (idle(red, status)) return;
    __shared__ cd sred[4][LDL_NB];
    __shared__ cd t[LDL_NB];
    __shared__ int last;
    const int b = j1 - j0;
    const int g = blockIdx.x, G = gridDim.x;
    const int r = threadIdx.x & 63, grp = threadIdx.x >> 6;
    const int c0 = j1 + g * chunk, c1 = min(n, c0 + chunk);
    cd s = mk(0.0, 0.0);
    if (r < b)
        for (int c = c0 + grp; c < c1; c += 4) s = cfma(ld2(A + (size_t)(j0 + r) + (size_t)c * ld), ldcg2(x + c), s);
    sred[grp][r] = s;
    __syncthreads();
    if (threadIdx.x < LDL_NB) {
        const cd v = (sred[0][r] + sred[1][r]) + (sred[2][r] + sred[3][r]);
        part[g * LDL_NB + r] = v;
    }
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) last = (atomicAdd(counter, 1) == G - 1);
    __syncthreads();
    if (!last) return;
    __threadfence();
    if (threadIdx.x < b) {
        cd q = mk(0.0, 0.0);
        for (int k = 0; k < G; k++) q = q + ldcg2(part + k * LDL_NB + threadIdx.x);
        t[threadIdx.x] = ld2(z + j0 + threadIdx.x) - q;
    }
    __syncthreads();
    if (threadIdx.x < b) {
        const int rr = threadIdx.x;
        cd v = mk(0.0, 0.0);
        for (int q = rr; q < b; q++) v = cfma(conj(ld2(linv + (size_t)(j0 + q) * LDL_NB + rr)), t[q], v);
        x[j0 + rr] = v;
    }
    if (threadIdx.x == 0) *counter = 0;
}

// ---------------------------------------------------------------------------
// Cooperative triangular solves: one CTA per LDL^H panel, all CTAs
// co-resident (cooperative launch).  CTA j accumulates the contributions of
// the panels it depends on in panel order, then applies its inverse diagonal
// block and publishes its own panel.  The neighbouring panel (j-1 forward,
// j+1 backward) is left out of that sum: its term is applied after the
// inverse block as one 64 x 64 product with the precomputed M_j = Linv_j
// U(j-1, j)^H or N_j = Linv_j^H U(j, j+1) (k_ldl_mn), so the step from one
// panel to the next is that product alone.
// The values are their own signal: the vector holds UNSET until a panel's
// CTA stores its 64 values, and a reader polls the values themselves (each
// 64-bit word is stored whole, and nothing else is read through them), so a
// step is a store and a load that sees it.  A flag beside the data costs a
// barrier, a release, the poll of the flag and then the load of the data:
// 2.3 us a step at K = 2000..4000 against 1.2 us.  Every wait is bounded:
// after SOLVE_SPIN_LIMIT polls, or as soon as any CTA has given up (the
// abort word), the CTA records ST_SOLVE_TIMEOUT and finishes without
// waiting; the host then reports the step as failed.
static_assert(SOLVE_SPIN_LIMIT == (1 << 22), "the default poll limit of the solves' waits");
// pitch of the 64 x 64 blocks in shared memory: 4 mod 8 double2, so that two
// rows' four columns fall on different banks
constexpr int LS_LD = LDL_NB + 4;

// Threads 0..63: the n <= 64 values at p into sv (zeros beyond), as they are
// computed; every thread returns whether they all were.
__device__ __forceinline__ bool wait_panel(const cd* p, int n, double2* sv, int* status, int* abort_word, int limit)
{
    bool ok = true;
    if (threadIdx.x < LDL_NB)
        sv[threadIdx.x] = (int)threadIdx.x < n ? wait_value(p + threadIdx.x, status, abort_word, limit, ok)
                                               : make_double2(0.0, 0.0);
    return __syncthreads_and(ok ? 1 : 0) != 0;
}

// Rows [j0, j0 + b) of a per-panel 64-column block (linv, lmf, lnb) into
// Ls[r][q] for q < bq, zeros elsewhere: asynchronous copies, all in flight at
// once (through registers the two blocks of a CTA took 4 us, a third of the
// whole solve at n = 201).
__device__ __forceinline__ void load_linv(const cd* __restrict__ linv, int j0, int b, double2* Ls, int bq = -1)
{
    if (bq < 0) bq = b;
    const int q = threadIdx.x & 63, r0 = threadIdx.x >> 6;
    const cd* src = linv + (size_t)(j0 + r0) * LDL_NB + q;
#pragma unroll 4
    for (int i = 0; i < 16; i++) {
        const int r = r0 + 4 * i;
        const bool in = r < b && q < bq;
        cp_async16(Ls + r * LS_LD + q, in ? src + (size_t)(4 * i) * LDL_NB : linv, in ? 16 : 0);
    }
    cp_async_commit();
}

// Row r = tid / 4 of the product of a 64 x 64 block in shared memory with
// the vector v: columns tid % 4, + 4, ..., summed over the four lanes, which
// all return it.
__device__ __forceinline__ cd row_product(const double2* __restrict__ B, const double2* __restrict__ v)
{
    const int r = threadIdx.x >> 2, q0 = threadIdx.x & 3;
    cd s0 = mk(0.0, 0.0), s1 = s0;
#pragma unroll
    for (int i = 0; i < 16; i += 2) {
        const double2 a = B[r * LS_LD + q0 + 4 * i], x = v[q0 + 4 * i];
        const double2 b = B[r * LS_LD + q0 + 4 * i + 4], y = v[q0 + 4 * i + 4];
        s0 = cfma(mk(a.x, a.y), mk(x.x, x.y), s0);
        s1 = cfma(mk(b.x, b.y), mk(y.x, y.y), s1);
    }
    cd s = s0 + s1;
#pragma unroll
    for (int o = 1; o <= 2; o <<= 1) {
        s.x += __shfl_xor_sync(0xffffffffu, s.x, o);
        s.y += __shfl_xor_sync(0xffffffffu, s.y, o);
    }
    return s;
}
// The same for the conjugate transpose of the block.
__device__ __forceinline__ cd row_product_h(const double2* __restrict__ B, const double2* __restrict__ v)
{
    const int r = threadIdx.x >> 2, q0 = threadIdx.x & 3;
    cd s = mk(0.0, 0.0);
#pragma unroll 4
    for (int i = 0; i < 16; i++) {
        const double2 a = B[(q0 + 4 * i) * LS_LD + r], x = v[q0 + 4 * i];
        s = cfma(mk(a.x, -a.y), mk(x.x, x.y), s);
    }
#pragma unroll
    for (int o = 1; o <= 2; o <<= 1) {
        s.x += __shfl_xor_sync(0xffffffffu, s.x, o);
        s.y += __shfl_xor_sync(0xffffffffu, s.y, o);
    }
    return s;
}

// Forward: y_j = Linv_j (w_j - sum_{a<j} U(a, j)^H y_a), z_j = invD_j y_j.
template <bool NEIGH>
__global__ void __launch_bounds__(256, NEIGH ? 1 : 2) k_fwd_coop(const cd* __restrict__ A, int ld, const int* __restrict__ bstart,
                                                  int nb, const cd* __restrict__ w, cd* __restrict__ y,
                                                  cd* __restrict__ z, const cd* __restrict__ invD,
                                                  const cd* __restrict__ linv, const cd* __restrict__ lmf,
                                                  int* status, int* abort_word, const double* __restrict__ idle_red)
{
    const bool off = idle_red && idle(idle_red, status);
    extern __shared__ double2 sm[];
    double2* Ls = sm;                          // Linv_j, [r][q]
    double2* Ms = sm + LDL_NB * LS_LD;         // NEIGH: M_j, [r][q]
    __shared__ double2 t[LDL_NB], ys[2][LDL_NB];
    const int j = blockIdx.x;
    const int j0 = bstart[j], j1 = bstart[j + 1], b = j1 - j0;
    const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5;
    load_linv(linv, j0, b, Ls);
    if (NEIGH && j > 0) load_linv(lmf, j0, b, Ms, j0 - bstart[j - 1]);
    if (off) {  // looked at while the blocks are on their way
        cp_async_wait<0>();
        return;
    }
    // this panel's right-hand side and pivots, read before the waits
    const int r = threadIdx.x >> 2;
    const cd wj = (threadIdx.x < b) ? ld2(w + j0 + threadIdx.x) : mk(0.0, 0.0);
    const cd dj = (r < b) ? ld2(invD + j0 + r) : mk(0.0, 0.0);
    // lane-partials for the 8 columns this warp owns
    cd acc[8];
#pragma unroll
    for (int m = 0; m < 8; m++) acc[m] = mk(0.0, 0.0);
    bool ok = true;
    const int limit = ((volatile int*)abort_word)[1];
    // every panel but the previous one; that one comes in below through
    // M_j = Linv_j U(j-1, j)^H
    const int alast = NEIGH ? j - 1 : j;
    // the factor block U(panel a, panel j) does not depend on panel a's
    // solution: it is loaded before the wait for that, with NEIGH (registers
    // of one CTA an SM) while the panel before it is still waited for
    auto load_u = [&](int a, cd (&u0)[8], cd (&u1)[8]) {
        const int a0 = bstart[a], a1 = bstart[a + 1];
        const int r0 = a0 + lane, r1 = a0 + lane + 32;
#pragma unroll
        for (int m = 0; m < 8; m++) {
            const int c = wp * 8 + m;
            const cd* col = A + (size_t)(j0 + c) * ld;
            u0[m] = (c < b && r0 < a1) ? ld2(col + r0) : mk(0.0, 0.0);
            u1[m] = (c < b && r1 < a1) ? ld2(col + r1) : mk(0.0, 0.0);
        }
    };
    auto apply = [&](int a, const cd (&u0)[8], const cd (&u1)[8]) {
        double2* sv = ys[a & 1];  // the other buffer may still be read
        ok = wait_panel(y + bstart[a], bstart[a + 1] - bstart[a], sv, status, abort_word, limit);
        const cd y0 = mk(sv[lane].x, sv[lane].y), y1 = mk(sv[lane + 32].x, sv[lane + 32].y);
#pragma unroll
        for (int m = 0; m < 8; m++) {
            acc[m] = cfma(conj(u0[m]), y0, acc[m]);
            acc[m] = cfma(conj(u1[m]), y1, acc[m]);
        }
    };
    cd ua[8], va[8];
    if (NEIGH) {
        cd ub[8], vb[8];
        if (alast > 0) load_u(0, ua, va);
        for (int a = 0; a < alast && ok; a += 2) {
            if (a + 1 < alast) load_u(a + 1, ub, vb);
            apply(a, ua, va);
            if (a + 1 < alast && ok) {
                if (a + 2 < alast) load_u(a + 2, ua, va);
                apply(a + 1, ub, vb);
            }
        }
    } else {
        for (int a = 0; a < alast && ok; a++) {
            load_u(a, ua, va);
            apply(a, ua, va);
        }
    }
    {
        double v[16];
#pragma unroll
        for (int m = 0; m < 8; m++) {
            v[2 * m] = acc[m].x;
            v[2 * m + 1] = acc[m].y;
        }
        const double sum = warp_transpose_sum<16>(v);
        if ((lane & 1) == 0) reinterpret_cast<double*>(t)[16 * wp + (lane >> 1)] = sum;
    }
    cp_async_wait<0>();
    __syncthreads();
    if (threadIdx.x < LDL_NB) t[threadIdx.x] = make_double2(wj.x - t[threadIdx.x].x, wj.y - t[threadIdx.x].y);
    __syncthreads();
    cd yr = row_product(Ls, t);
    if (NEIGH && j > 0) {
        // y_j -= M_j y_{j-1}
        double2* sv = ys[(j - 1) & 1];
        if (ok && wait_panel(y + bstart[j - 1], j0 - bstart[j - 1], sv, status, abort_word, limit)) yr = yr - row_product(Ms, sv);
    }
    if ((threadIdx.x & 3) == 0 && r < b) {
        y[j0 + r] = yr;
        z[j0 + r] = cmul(yr, dj);
    }
}

// Backward: x_j = Linv_j^H (z_j - sum_{c>j} U(j, c) x_c).
template <bool NEIGH>
__global__ void __launch_bounds__(256, NEIGH ? 1 : 2) k_bwd_coop(const cd* __restrict__ A, int ld, const int* __restrict__ bstart,
                                                  int nb, const cd* __restrict__ z, cd* __restrict__ x,
                                                  const cd* __restrict__ linv, const cd* __restrict__ lnb,
                                                  int* status, int* abort_word, const double* __restrict__ idle_red)
{
    const bool off = idle(idle_red, status);
    extern __shared__ double2 sm[];
    double2* Ls = sm;
    double2* red = sm + LDL_NB * LS_LD;  // [8][64] warp partials
    double2* Ns = red + 8 * LDL_NB;      // NEIGH: N_j, [r][q]
    __shared__ double2 t[LDL_NB], xs[2][LDL_NB];
    const int j = blockIdx.x;
    const int j0 = bstart[j], j1 = bstart[j + 1], b = j1 - j0;
    const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5;
    load_linv(linv, j0, b, Ls);
    if (NEIGH && j + 1 < nb) load_linv(lnb, j0, b, Ns, bstart[j + 2] - j1);
    if (off) {
        cp_async_wait<0>();
        return;
    }
    const int r = threadIdx.x >> 2;
    const cd zj = (threadIdx.x < b) ? ld2(z + j0 + threadIdx.x) : mk(0.0, 0.0);  // read before the waits
    cd a0 = mk(0.0, 0.0), a1 = mk(0.0, 0.0);  // rows lane, lane + 32
    bool ok = true;
    const int limit = ((volatile int*)abort_word)[1];
    // every later panel but the next one; that one comes in below through
    // N_j = Linv_j^H U(j, j+1)
    const int clast = NEIGH ? j + 1 : j;
    auto load_u = [&](int c, cd (&u0)[8], cd (&u1)[8]) {
        const int c0 = bstart[c], c1 = bstart[c + 1];
#pragma unroll
        for (int i = 0; i < 8; i++) {
            const int col = c0 + wp + 8 * i;
            const cd* u = A + (size_t)col * ld + j0;
            u0[i] = (col < c1 && lane < b) ? ld2(u + lane) : mk(0.0, 0.0);
            u1[i] = (col < c1 && lane + 32 < b) ? ld2(u + lane + 32) : mk(0.0, 0.0);
        }
    };
    auto apply = [&](int c, const cd (&u0)[8], const cd (&u1)[8]) {
        double2* sv = xs[c & 1];
        ok = wait_panel(x + bstart[c], bstart[c + 1] - bstart[c], sv, status, abort_word, limit);
#pragma unroll
        for (int i = 0; i < 8; i++) {
            const double2 v = sv[wp + 8 * i];
            a0 = cfma(u0[i], mk(v.x, v.y), a0);
            a1 = cfma(u1[i], mk(v.x, v.y), a1);
        }
    };
    cd ua[8], va[8];
    if (NEIGH) {
        cd ub[8], vb[8];
        if (nb - 1 > clast) load_u(nb - 1, ua, va);
        for (int c = nb - 1; c > clast && ok; c -= 2) {
            if (c - 1 > clast) load_u(c - 1, ub, vb);
            apply(c, ua, va);
            if (c - 1 > clast && ok) {
                if (c - 2 > clast) load_u(c - 2, ua, va);
                apply(c - 1, ub, vb);
            }
        }
    } else {
        for (int c = nb - 1; c > clast && ok; c--) {
            load_u(c, ua, va);
            apply(c, ua, va);
        }
    }
    red[wp * LDL_NB + lane] = make_double2(a0.x, a0.y);
    red[wp * LDL_NB + lane + 32] = make_double2(a1.x, a1.y);
    cp_async_wait<0>();
    __syncthreads();
    if (threadIdx.x < LDL_NB) {
        cd s = mk(0.0, 0.0);
#pragma unroll
        for (int q = 0; q < 8; q++) s = s + mk(red[q * LDL_NB + threadIdx.x].x, red[q * LDL_NB + threadIdx.x].y);
        t[threadIdx.x] = make_double2(zj.x - s.x, zj.y - s.y);
    }
    __syncthreads();
    cd xr = row_product_h(Ls, t);
    if (NEIGH && j + 1 < nb) {
        // x_j -= N_j x_{j+1}
        double2* sv = xs[(j + 1) & 1];
        if (ok && wait_panel(x + bstart[j + 1], bstart[j + 2] - bstart[j + 1], sv, status, abort_word, limit))
            xr = xr - row_product(Ns, sv);
    }
    if ((threadIdx.x & 3) == 0 && r < b) x[j0 + r] = xr;
}

// Block-wide deterministic sums (1024 threads).
template <int NV>
__device__ __forceinline__ void block_sum(double (&v)[NV], double* sh)
{
    const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5;
#pragma unroll
    for (int k = 0; k < NV; k++)
#pragma unroll
        for (int o = 16; o >= 1; o >>= 1) v[k] += __shfl_xor_sync(0xffffffffu, v[k], o);
    __syncthreads();
    if (lane == 0)
#pragma unroll
        for (int k = 0; k < NV; k++) sh[wp * NV + k] = v[k];
    __syncthreads();
#pragma unroll
    for (int k = 0; k < NV; k++) {
        double s = 0.0;
        for (int q = 0; q < 32; q++) s += sh[q * NV + k];
        v[k] = s;
    }
}

// Normalisation, convergence measure and convergence of one step from the
// solution xw (src/linalg.f90:1894-1908); ends with v <- x.
__global__ void __launch_bounds__(1024) k_iter_norm(int n, const cd* __restrict__ xw, cd* __restrict__ x,
                                                    cd* __restrict__ v, double sqrtn, double tol,
                                                    double* __restrict__ red, const int* __restrict__ status)
{
    if (idle(red, status)) return;
    __shared__ double sh[32 * 3];
    __shared__ double smax[32];
    const int tid = threadIdx.x, lane = tid & 31, wp = tid >> 5;
    double m = 0.0;
    for (int j = tid; j < n; j += 1024) {
        const cd a = xw[j];
        m = fmax(m, fmax(fabs(a.x), fabs(a.y)));
    }
#pragma unroll
    for (int o = 16; o >= 1; o >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
    if (lane == 0) smax[wp] = m;
    __syncthreads();
    double t1 = 0.0;
    for (int q = 0; q < 32; q++) t1 = fmax(t1, smax[q]);
    const double ra = 1.0 / t1;
    double acc[3] = {0.0, 0.0, 0.0};
    for (int j = tid; j < n; j += 1024) {
        cd a = xw[j];
        a = cd{ra * a.x, ra * a.y};
        x[j] = a;
        const cd b = v[j];
        acc[0] = fma(a.x, b.x, fma(a.y, b.y, acc[0]));   // Re conj(x) v
        acc[1] = fma(a.x, b.y, fma(-a.y, b.x, acc[1]));  // Im conj(x) v
        acc[2] = fma(b.x, b.x, fma(b.y, b.y, acc[2]));
    }
    block_sum<3>(acc, sh);
    const cd tc = cd{acc[0] / acc[2], acc[1] / acc[2]};
    double d[1] = {0.0};
    for (int j = tid; j < n; j += 1024) {
        const cd a = x[j];
        const cd s = cfms(tc, v[j], a);
        d[0] = fma(s.x, s.x, fma(s.y, s.y, d[0]));
    }
    __syncthreads();
    block_sum<1>(d, sh);
    if (tid == 0) {
        const double nd = sqrtn * sqrt(d[0]), it = red[RD_ITERS];
        const double prev = it > 0.0 ? red[RD_NORMDIFF] : DBL_MAX;
        red[RD_NORMDIFF] = nd;
        red[RD_ITERS] = it + 1.0;
        red[RD_GAIN] = nd / prev;
        red[RD_DONE] = (tol > 0.0 ? nd <= tol : (nd > prev && nd <= fabs(tol))) ? 1.0 : 0.0;
    }
    __syncthreads();
    for (int j = tid; j < n; j += 1024) v[j] = x[j];
}

// Per-column terms of x^H A x over the lower triangle (VMMHMV,
// src/linalg.f90:1195-1206) for A = B (blockIdx.y = 0) and A = M (1).
__global__ void __launch_bounds__(256) k_vmm_cols(const cd* __restrict__ B, const cd* __restrict__ M, int ld, int n,
                                                  const cd* __restrict__ x, double* __restrict__ colval,
                                                  const double* __restrict__ red, const int* __restrict__ status, int always)
{
    if (idle_rayleigh(red, status, always)) return;
    const int k = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (k >= n) return;
    const cd* A = (blockIdx.y == 0) ? B : M;
    const cd* col = A + (size_t)k * ld;
    double sr = 0.0, si = 0.0;
    for (int j = k + 1 + lane; j < n; j += 32) {
        const cd a = ld2(col + j), xj = ld2(x + j);
        sr = fma(xj.x, a.x, fma(xj.y, a.y, sr));
        si = fma(xj.y, a.x, fma(-xj.x, a.y, si));
    }
#pragma unroll
    for (int o = 16; o >= 1; o >>= 1) {
        sr += __shfl_xor_sync(0xffffffffu, sr, o);
        si += __shfl_xor_sync(0xffffffffu, si, o);
    }
    if (lane == 0) {
        const cd xk = ld2(x + k);
        const double dk = ld2(col + k).x;
        colval[(size_t)blockIdx.y * n + k] = fma(xk.x * xk.x + xk.y * xk.y, dk, 2.0 * (xk.x * sr + xk.y * si));
    }
}

// The three quadratic forms; x is then scaled to x^H B x = 1 (specif_norm 0)
// or x^H x = 1 (1).
__global__ void __launch_bounds__(1024) k_vmm_reduce(int n, const double* __restrict__ colval, cd* __restrict__ x,
                                                     double* __restrict__ red, const int* __restrict__ status, int always,
                                                     int specif_norm)
{
    __shared__ double sh[32 * 3];
    if (idle_rayleigh(red, status, always)) return;
    double acc[3] = {0.0, 0.0, 0.0};
    for (int j = threadIdx.x; j < n; j += 1024) {
        acc[0] += colval[j];
        acc[1] += colval[n + j];
        const cd a = x[j];
        acc[2] = fma(a.x, a.x, fma(a.y, a.y, acc[2]));
    }
    block_sum<3>(acc, sh);
    if (threadIdx.x == 0) {
        red[RD_T1] = acc[0];
        red[RD_T2] = acc[1];
        red[RD_XX] = acc[2];
    }
    if (specif_norm != 0 && specif_norm != 1) return;
    const double f = 1.0 / sqrt(specif_norm == 0 ? acc[0] : acc[2]);
    for (int j = threadIdx.x; j < n; j += 1024) {
        const cd a = x[j];
        x[j] = cd{a.x * f, a.y * f};
    }
}

// ---------------------------------------------------------------------------
// Shared memory of the cooperative solves: the inverse diagonal block, the
// partial sums and, with NEIGH, the neighbour product M_j / N_j.
static size_t coop_smem(bool neigh)
{
    return (size_t)(LDL_NB * LS_LD + 8 * LDL_NB + (neigh ? LDL_NB * LS_LD : 0)) * sizeof(double2);
}

template <bool NEIGH>
static int coop_blocks(int dev)
{
    const int sm = (int)coop_smem(NEIGH);
    cudaFuncSetAttribute(k_fwd_coop<NEIGH>, cudaFuncAttributeMaxDynamicSharedMemorySize, sm);
    cudaFuncSetAttribute(k_bwd_coop<NEIGH>, cudaFuncAttributeMaxDynamicSharedMemorySize, sm);
    int coop = 0, nsm = 0, per1 = 0, per2 = 0;
    cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev);
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per1, k_fwd_coop<NEIGH>, 256, sm);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per2, k_bwd_coop<NEIGH>, 256, sm);
    cudaGetLastError();
    return coop ? nsm * std::min(per1, per2) : -1;
}

// Largest grid the cooperative solves may use on this device (-1: none),
// without and with the neighbour products.
static int coop_capacity(Ctx& c, bool neigh)
{
    if (!c.coop_max_blocks) {
        c.coop_max_blocks = coop_blocks<false>(c.dev);
        c.coop_max_neigh = coop_blocks<true>(c.dev);
    }
    return neigh ? c.coop_max_neigh : c.coop_max_blocks;
}

static int solve_multi_launch(Ctx& c, int n)
{
    const int nb = (int)c.blk_start.size();
    for (int i = 0; i < nb; i++) {
        const int j0 = c.blk_start[i], j1 = (i + 1 < nb) ? c.blk_start[i + 1] : n;
        int G = (j0 + 127) / 128;
        G = G < 1 ? 1 : (G > SOLVE_G_MAX ? SOLVE_G_MAX : G);
        const int chunk = (j0 + G - 1) / G;
        k_fwd<<<G, 256, 0, c.stream>>>(c.F, c.ld, j0, j1, chunk > 0 ? chunk : 1, c.w, c.yv, c.zv, c.invD, c.linv,
                                      c.spart, c.counters, c.red, c.status);
        c.launches++;
    }
    for (int i = nb - 1; i >= 0; i--) {
        const int j0 = c.blk_start[i], j1 = (i + 1 < nb) ? c.blk_start[i + 1] : n;
        const int rest = n - j1;
        int G = (rest + 127) / 128;
        G = G < 1 ? 1 : (G > SOLVE_G_MAX ? SOLVE_G_MAX : G);
        const int chunk = (rest + G - 1) / G;
        k_bwd<<<G, 256, 0, c.stream>>>(c.F, c.ld, j0, j1, n, chunk > 0 ? chunk : 1, c.zv, c.xw, c.linv, c.spart,
                                      c.counters + 1, c.red, c.status);
        c.launches++;
    }
    return 0;
}

// ---------------------------------------------------------------------------
// The bordered step of LDLHF for one new row (src/linalg.f90:356-391 with
// m = n): column m0 of L^H is U(:, m0) = invD o a with a = L0^-1 M(:, m0),
// one forward solve with the existing factor, and the pivot d = M(m0, m0) -
// sum_q conj(a_q) U(q, m0).  At K = 2001: 70 us in three launches; a panel
// solve and a rank-64 update of the one column per existing panel took 567
// us in 64.
// ---------------------------------------------------------------------------

// w = M(0..m0-1, m0) from the row that holds its conjugate; y as the solve
// wants it.
__global__ void __launch_bounds__(256) k_border_rhs(const cd* __restrict__ A, int ld, int m0, cd* __restrict__ w,
                                                    cd* __restrict__ y)
{
    const int r = blockIdx.x * 256 + threadIdx.x;
    if (r >= m0) return;
    w[r] = conj(A[(size_t)m0 + (size_t)r * ld]);
    y[r] = unset();
}

// The column, the pivot (its imaginary part kept with cplx, as the reference
// keeps it) and the one-row panel's blocks for the solves: Linv = 1, M of the
// new panel and N of the last existing one (rows [p0, m0)).
__global__ void __launch_bounds__(1024) k_border_finish(cd* __restrict__ A, int ld, int m0, int p0,
                                                        const cd* __restrict__ y, const cd* __restrict__ z,
                                                        cd* __restrict__ invD, cd* __restrict__ linv,
                                                        cd* __restrict__ lmf, cd* __restrict__ lnb,
                                                        int* __restrict__ status, int cplx)
{
    __shared__ double sh[32 * 2];
    const int tid = threadIdx.x;
    double acc[2] = {0.0, 0.0};
    for (int q = tid; q < m0; q += 1024) {
        const cd u = z[q], s = cmul(conj(y[q]), u);
        acc[0] += s.x;
        acc[1] += s.y;
        A[(size_t)q + (size_t)m0 * ld] = u;
    }
    block_sum<2>(acc, sh);
    const int bp = m0 - p0;
    if (tid == 0) {
        const double xr = A[(size_t)m0 + (size_t)m0 * ld].x - acc[0], xi = cplx ? acc[1] : 0.0;
        cd id = mk(0.0, 0.0);
        if (xr == 0.0 && xi == 0.0)
            atomicCAS(status + ST_ZERO_PIVOT, 0, m0 + 1);
        else
            id = cplx ? crcp(mk(xr, xi)) : mk(1.0 / xr, 0.0);
        invD[m0] = id;
    }
    if (tid < LDL_NB) {
        linv[(size_t)m0 * LDL_NB + tid] = mk(tid == 0 ? 1.0 : 0.0, 0.0);
        lmf[(size_t)m0 * LDL_NB + tid] = tid < bp ? conj(z[p0 + tid]) : mk(0.0, 0.0);
    }
    // N(r, 0) = sum_q conj(Linv(q, r)) U(p0 + q, m0), four lanes a row
    const int r = (tid >> 2) & 63;
    if (tid < 4 * LDL_NB) {
        cd s = mk(0.0, 0.0);
        if (r < bp)
            for (int q = r + (tid & 3); q < bp; q += 4)
                s = cfma(conj(ld2(linv + (size_t)(p0 + q) * LDL_NB + r)), z[p0 + q], s);
#pragma unroll
        for (int o = 1; o <= 2; o <<= 1) {
            s.x += __shfl_xor_sync(0xffffffffu, s.x, o);
            s.y += __shfl_xor_sync(0xffffffffu, s.y, o);
        }
        if (r < bp)
            for (int q = tid & 3; q < LDL_NB; q += 4)
                lnb[(size_t)(p0 + r) * LDL_NB + q] = q == 0 ? s : mk(0.0, 0.0);
    }
}

// red: the iteration's state, or null outside it.
static int launch_fwd(Ctx& c, int nb, bool neigh, const double* red)
{
    const size_t sm = coop_smem(neigh);
    int* abort_word = c.counters + 2;
    const int* bs = c.dblk;
    const cd *H = c.F, *w = c.w, *invD = c.invD, *linv = c.linv, *lmf = c.lmf;
    int ld = c.ld;
    void* args[] = {(void*)&H, &ld, (void*)&bs, &nb, (void*)&w, &c.yv, &c.zv, (void*)&invD, (void*)&linv, (void*)&lmf,
                    &c.status, &abort_word, (void*)&red};
    const void* k = neigh ? (const void*)k_fwd_coop<true> : (const void*)k_fwd_coop<false>;
    if (cudaLaunchCooperativeKernel(k, nb, 256, args, sm, c.stream) != cudaSuccess) return -2;
    c.launches++;
    return 0;
}

static int solve_cooperative(Ctx& c, bool neigh)
{
    int nb = (int)c.blk_start.size();
    const double* red = c.red;
    const int r = launch_fwd(c, nb, neigh, red);
    if (r) return r;
    int* abort_word = c.counters + 2;
    const int* bs = c.dblk;
    const cd *H = c.F, *linv = c.linv, *lnb = c.lnb, *zv = c.zv;
    int ld = c.ld;
    void* args[] = {(void*)&H, &ld, (void*)&bs, &nb, (void*)&zv, &c.xw, (void*)&linv, (void*)&lnb,
                    &c.status, &abort_word, (void*)&red};
    const void* k = neigh ? (const void*)k_bwd_coop<true> : (const void*)k_bwd_coop<false>;
    if (cudaLaunchCooperativeKernel(k, nb, 256, args, coop_smem(neigh), c.stream) != cudaSuccess) return -2;
    c.launches++;
    return 0;
}

// Row m0 beside the factor of rows 0..m0-1, whose nexist panels (the last
// one truncated at m0) are in c.dblk.  1: not available for so many panels.
int border_row(Ctx& c, int m0, int nexist)
{
    const bool neigh = nexist <= coop_capacity(c, true);
    if (nexist < 1 || (!neigh && nexist > coop_capacity(c, false))) return 1;
    k_border_rhs<<<(m0 + 255) / 256, 256, 0, c.stream>>>(c.F, c.ld, m0, c.w, c.yv);
    if (cudaMemsetAsync(c.counters + 2, 0, sizeof(int), c.stream) != cudaSuccess) return -2;  // the abort word
    const int r = launch_fwd(c, nexist, neigh, nullptr);
    if (r) return r;
    int p0 = 0;  // first row of the last existing panel
    for (int s : c.blk_start)
        if (s < m0) p0 = s;
    k_border_finish<<<1, 1024, 0, c.stream>>>(c.F, c.ld, m0, p0, c.yv, c.zv, c.invD, c.linv, c.lmf, c.lnb, c.status,
                                              c.pivot_mode);
    c.launches += 2;
    return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

// Whether a step is a launch per panel: more panels than co-resident CTAs.
bool invit_by_panels(Ctx& c) { return (int)c.blk_start.size() > coop_capacity(c, false); }

int invit_step(Ctx& c, int n, double tol)
{
    k_hemv<<<(n * 32 + 255) / 256, 256, 0, c.stream>>>(c.S, c.ld, n, c.c, c.w, c.yv, c.xw, c.red, c.status);
    c.launches++;
    const int nb = (int)c.blk_start.size();
    // the neighbour products take a second 64 x 64 block of shared memory
    // (one CTA per SM): used while every panel still has an SM of its own
    int r;
    if (nb <= coop_capacity(c, true))
        r = solve_cooperative(c, true);
    else if (!invit_by_panels(c))
        r = solve_cooperative(c, false);
    else
        r = solve_multi_launch(c, n);
    if (r) return r;
    k_iter_norm<<<1, 1024, 0, c.stream>>>(n, c.xw, c.x, c.c, sqrt(2.0 * n), tol, c.red, c.status);
    c.launches++;
    return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

// Once the iteration has converged, or `always`.
int invit_rayleigh(Ctx& c, int n, bool always, int specif_norm)
{
    dim3 g((n * 32 + 255) / 256, 2);
    k_vmm_cols<<<g, 256, 0, c.stream>>>(c.S, c.F, c.ld, n, c.x, c.colval, c.red, c.status, always);
    k_vmm_reduce<<<1, 1024, 0, c.stream>>>(n, c.colval, c.x, c.red, c.status, always, specif_norm);
    c.launches += 2;
    return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

}  // namespace ecg
