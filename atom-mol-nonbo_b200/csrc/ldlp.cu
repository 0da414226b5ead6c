// ldlp.cu -- LDL^H factorisation of a whole matrix (no existing rows) as one
// persistent cooperative kernel over 64 x 64 tiles, the drop-in for LDLHF
// with m = 1 (src/linalg.f90:316-455).
//
// Same storage contract and recurrence as ldlh.cu: M's lower triangle is left
// untouched, the strict upper triangle receives L^H, invD receives 1/d; the
// working Schur complement W(r, c), r < c, lives in the upper triangle and
// its diagonal in dw.  The factorisation is split into tasks on 64 x 64 tiles
// (R, C), R <= C, of panel index s:
//   D(s)        eliminate the diagonal tile (s, s): U_ss, L_ss^-1 (also what
//               the triangular solves need), invD, pivots d_s (written to dw
//               over the consumed working diagonal);
//   T(s, C)     panel rows of tile (s, C): U(s, C) = invD L_ss^-1 W(s, C);
//   B(s, R, C)  W(R, C) -= conj(U(s, R))^T diag(d_s) U(s, C), s < R <= C
//               (the unscaled rows of the reference's recurrence, d U, are
//               formed in registers from U and d instead of being stored).
// Every tile has a counter: the number of panels applied to it (D and T set
// it to s + 1 when the tile is final).  A task waits (bounded) until its
// tiles carry the counts it needs:
//   D(s): cnt(s,s) >= s;  T(s,C): cnt(s,s) >= s+1, cnt(s,C) >= s;
//   B(s,R,C): cnt(s,R) >= s+1, cnt(s,C) >= s+1, cnt(R,C) >= s.
// CTA 0, alone on its SM, runs the chain D(s) -> T(s, s+1) -> B(s, s+1,
// s+1) -> D(s+1) with the diagonal tile kept in registers.  The other
// CTAs (all co-resident: cooperative launch) take every other task from a
// list in a fixed order through one atomic counter; updates far from their
// panels are one task for four of them, and a nearer one whose group's next
// panels are already final applies them too (rank up to 256).  The list is
// a topological order of the dependency graph, made on the host by list
// scheduling on as many simulated workers as the grid has CTAs, always
// starting the ready task with the longest remaining path (upward rank).
// Because every task's dependencies come earlier in that order (the chain's
// included) and every CTA is resident, the earliest unfinished task can
// always proceed: the kernel cannot deadlock.  Waits are still bounded (the
// poll limit of ecg_set_wait_limit); a CTA that gives up records
// ST_SOLVE_TIMEOUT and sets the abort word, after which every CTA stops
// taking tasks.
//
// What bounds it: the FP64 tensor cores for the list (37 TFLOP/s; DFMA and
// DMMA share that unit), the chain's latency where few panels are left.  On a
// B200 the chain takes 32 us a panel (D 18, T 9, B 4 and a part overlapped
// with D; 47 us with an elimination through shared memory and substitution
// in T), and the list's updates run at 95 % of the tensor cores, so whole
// factorisations take 0.31 ms at K = 500 (0.46 before both), 0.88 at 1500
// (1.24), 3.63 at 4000 (4.94), 45.5 at 10000 (57.2 per panel step).  Two CTAs an SM take 217 KB of
// shared memory and leave about 28 KB of L1, so a spilled register comes back
// from L2: the chain with 200 bytes of stack ran D(s) in 32 us, with 32 bytes
// in 18.  Every array of the chain is sized to stay within 128 registers.
#include <algorithm>
#include <queue>
#include <utility>
#include <vector>
#include "ecg_internal.h"
#include "zmma.cuh"
#include "tma_ring.cuh"

namespace ecg {

constexpr unsigned LP_D = 0, LP_T = 1, LP_B = 2;
constexpr unsigned LP_NONE = 0xffffffffu;
constexpr int LP_OP = TMA_KC * LDL_NB;  // double2 of one staged operand (8 KB)
constexpr int LP_MERGE = 4;        // most panels one trailing update applies at once
// Aligned groups of LP_MERGE panels whose update of a tile row at least this
// far from the group's first panel is one task of the list: nearer rows are
// wanted before the group's last panel is there.
constexpr int LP_FAR = 8;
// 1 KB to align the stages, which the swizzle wants
constexpr size_t LP_SMEM_B = 1024 + (size_t)(TMA_ST * 2 * LP_OP + LP_MERGE * LDL_NB) * sizeof(double2);

__host__ __device__ __forceinline__ unsigned lp_code(unsigned type, int s, int R, int C, unsigned half = 0)
{
    return type << 30 | half << 29 | (unsigned)s << 20 | (unsigned)R << 10 | (unsigned)C;
}
// The updates of the two tile rows after panel s (the band the diagonal
// chain waits on), except the chain's own B(s, s+1, s+1), run as two tasks
// on the column halves of the tile, so each takes half the time on its SM.
__host__ __device__ __forceinline__ bool lp_split(int s, int R, int C)
{
    return R <= s + 2 && !(R == s + 1 && C == s + 1);
}
// One list task for panels s..s+LP_MERGE-1 on tile (R, C) (s a multiple of
// LP_MERGE); its code has the half bit, which whole updates do not use.
__host__ __device__ __forceinline__ bool lp_grouped(int s, int R)
{
    return R >= s - s % LP_MERGE + LP_FAR;
}
// counter of tile (R, C), R <= C: column-wise packed triangle
__host__ __device__ __forceinline__ long long lp_tix(int R, int C) { return (long long)C * (C + 1) / 2 + R; }

// ---------------------------------------------------------------------------
// Host: the task list.
// ---------------------------------------------------------------------------
// Task weights (us) for the list scheduler: the time a CTA is held by a
// task on a B200 with two CTAs per SM, waits and merged updates included
// (globaltimer records of ecg_factor_trace); a split update counts half.
// Only the ratios matter.  Measured for g (ms at K = 2500, 4000, 9000):
// 75 1.62, 3.81, 33.5; 140 1.59, 3.61, 33.3; 180 1.55, 3.63, 33.2; 320
// 1.55, 3.74, 33.3.  Per-panel tasks in place of groups: 1.52, 3.79, 34.9.
struct LpCost {
    double d = 21.0, t = 40.0, b = 60.0, bd = 40.0, g = 180.0;  // g: one task for LP_MERGE panels
};

// Tasks of a factorisation with np panels: the list the P CTAs other than
// the chain CTA take, and (if full is given) every task in the simulated
// start order, the chain's included.  With `group` the far updates are one
// task for LP_MERGE panels: found merged one by one at run time they left
// 440,000 empty tasks at K = 10000, and the list took the host 290 ms.
static void lp_schedule(int np, int P, const LpCost& cost, bool group, std::vector<unsigned>& list,
                        std::vector<unsigned>* full = nullptr)
{
    std::vector<unsigned> code;
    std::vector<int> idD(np);
    std::vector<int> idT((size_t)np * np, -1);
    std::vector<int> idB((size_t)np * np * np, -1);  // first node of B(s, R, C)
    auto bix = [&](int s, int R, int C) -> size_t { return ((size_t)s * np + R) * np + C; };
    for (int s = 0; s < np; s++) {
        idD[s] = (int)code.size();
        code.push_back(lp_code(LP_D, s, s, s));
        for (int C = s + 1; C < np; C++) {
            idT[(size_t)s * np + C] = (int)code.size();
            code.push_back(lp_code(LP_T, s, s, C));
        }
        for (int R = s + 1; R < np; R++)
            for (int C = R; C < np; C++) {
                if (group && lp_grouped(s, R)) {  // created with the group's last panel
                    if (s % LP_MERGE == LP_MERGE - 1) {
                        idB[bix(s, R, C)] = (int)code.size();
                        code.push_back(lp_code(LP_B, s - s % LP_MERGE, R, C, 1));
                    }
                    continue;
                }
                idB[bix(s, R, C)] = (int)code.size();
                code.push_back(lp_code(LP_B, s, R, C));
                if (lp_split(s, R, C)) code.push_back(lp_code(LP_B, s, R, C, 1));  // the second column half
            }
    }
    const int N = (int)code.size();
    // predecessors in creation order, which is topological: an update that
    // is split in two column halves counts as both halves
    constexpr int NPRED = 6;
    std::vector<int> pred((size_t)N * NPRED, -1);
    std::vector<double> w((size_t)N);
    for (int t = 0; t < N; t++) {
        const unsigned c = code[t];
        const int type = c >> 30, s = (c >> 20) & 511, R = (c >> 10) & 1023, C = c & 1023;
        int* p = &pred[(size_t)t * NPRED];
        int k = 0;
        auto addB = [&](int s2, int R2, int C2) {
            const int b = idB[bix(s2, R2, C2)];
            p[k++] = b;
            if (lp_split(s2, R2, C2)) p[k++] = b + 1;
        };
        if (type == LP_D) {
            if (s > 0) addB(s - 1, s, s);
            w[t] = cost.d;
        } else if (type == LP_T) {
            p[k++] = idD[s];
            if (s > 0) addB(s - 1, s, C);
            w[t] = cost.t;
        } else {
            const bool g = group && lp_grouped(s, R);
            const int last = g ? s + LP_MERGE - 1 : s;
            p[k++] = idT[(size_t)last * np + R];
            if (C != R) p[k++] = idT[(size_t)last * np + C];
            if (s > 0) addB(s - 1, R, C);
            w[t] = g ? cost.g : ((R == C) ? cost.bd : cost.b) * (lp_split(s, R, C) ? 0.5 : 1.0);
        }
    }
    // successors (CSR)
    std::vector<int> so((size_t)N + 1, 0), sl;
    for (int t = 0; t < N; t++)
        for (int k = 0; k < NPRED; k++)
            if (pred[(size_t)t * NPRED + k] >= 0) so[(size_t)pred[(size_t)t * NPRED + k] + 1]++;
    for (int t = 0; t < N; t++) so[(size_t)t + 1] += so[(size_t)t];
    sl.resize((size_t)so[(size_t)N]);
    {
        std::vector<int> fill(so.begin(), so.end() - 1);
        for (int t = 0; t < N; t++)
            for (int k = 0; k < NPRED; k++) {
                const int p = pred[(size_t)t * NPRED + k];
                if (p >= 0) sl[(size_t)fill[(size_t)p]++] = t;
            }
    }
    // upward rank: own duration plus the longest path through the successors
    std::vector<double> rank((size_t)N);
    for (int t = N - 1; t >= 0; t--) {
        double m = 0.0;
        for (int e = so[(size_t)t]; e < so[(size_t)t + 1]; e++) m = std::max(m, rank[(size_t)sl[(size_t)e]]);
        rank[(size_t)t] = w[(size_t)t] + m;
    }
    // list scheduling: the chain worker runs D(s), T(s, s+1), B(s, s+1,
    // s+1) in that order, each as soon as it is ready; the P list workers
    // start the ready task of highest rank (earliest created among equals)
    // whenever one of them is free.  `full` receives every task in start
    // order.
    std::vector<char> pool((size_t)N, 1);  // 0 chain, 1 list
    std::vector<int> cseq;
    for (int s = 0; s < np; s++) {
        pool[(size_t)idD[s]] = 0;
        cseq.push_back(idD[s]);
        if (s + 1 < np) {
            const int t = idT[(size_t)s * np + s + 1], b = idB[bix(s, s + 1, s + 1)];
            pool[(size_t)t] = pool[(size_t)b] = 0;
            cseq.push_back(t);
            cseq.push_back(b);
        }
    }
    std::vector<int> npred((size_t)N, 0);
    for (int t = 0; t < N; t++)
        for (int k = 0; k < NPRED; k++) npred[(size_t)t] += pred[(size_t)t * NPRED + k] >= 0;
    typedef std::pair<double, int> Item;
    std::priority_queue<Item> ready;                                        // (rank, -id)
    std::priority_queue<Item, std::vector<Item>, std::greater<Item>> busy;  // (finish, id)
    for (int t = 0; t < N; t++)
        if (npred[(size_t)t] == 0 && pool[(size_t)t]) ready.push({rank[(size_t)t], -t});
    list.clear();
    if (full) {
        full->clear();
        full->reserve((size_t)N);
    }
    int free_w[2] = {1, std::max(1, P)};
    size_t ci = 0;
    int started = 0;
    double now = 0.0;
    while (started < N) {
        if (free_w[0] > 0 && ci < cseq.size() && npred[(size_t)cseq[ci]] == 0) {
            const int t = cseq[ci];
            if (full) full->push_back(code[(size_t)t]);
            busy.push({now + w[(size_t)t], t});
            free_w[0]--;
            started++;
        }
        while (free_w[1] > 0 && !ready.empty()) {
            const int t = -ready.top().second;
            ready.pop();
            list.push_back(code[(size_t)t]);
            if (full) full->push_back(code[(size_t)t]);
            busy.push({now + w[(size_t)t], t});
            free_w[1]--;
            started++;
        }
        if (busy.empty()) break;  // cannot happen for a valid graph
        const Item f = busy.top();
        busy.pop();
        now = f.first;
        const int fp = pool[(size_t)f.second];
        free_w[fp]++;
        if (fp == 0) ci++;
        for (int e = so[(size_t)f.second]; e < so[(size_t)f.second + 1]; e++) {
            const int q = sl[(size_t)e];
            if (--npred[(size_t)q] == 0 && pool[(size_t)q]) ready.push({rank[(size_t)q], -q});
        }
    }
}

// ---------------------------------------------------------------------------
// Device.
// ---------------------------------------------------------------------------
__device__ __forceinline__ unsigned lp_ld_acquire(const unsigned* p)
{
    unsigned v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void lp_st_release(unsigned* p, unsigned v)
{
    asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ double2 lp_ldcg(const cd* p) { return __ldcg(reinterpret_cast<const double2*>(p)); }
__device__ __forceinline__ void lp_mma(double& c0, double& c1, double a, double b)
{
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
                 : "+d"(c0), "+d"(c1)
                 : "d"(a), "d"(b));
}
__device__ __forceinline__ cd lp_shfl(cd v, int src)
{
    return cd{__shfl_sync(0xffffffffu, v.x, src), __shfl_sync(0xffffffffu, v.y, src)};
}

// T(s, C): U(s, C) = invD Linv_ss W(s, C) for the 64 columns of tile (s, C),
// Linv_ss = L_ss^-1 (unit lower) as the diagonal task left it: one product
// with a triangular matrix on the FP64 tensor cores, 288 independent-ordered
// mma a warp and no step that waits for another.  (Substitution by 8-row
// blocks, the form before, is a chain of eight dependent steps through
// shared memory: 23.4 us a task with two CTAs an SM at K = 4000, 12.4 us on
// the chain's own SM.)
// Linv_ss sits in shared memory as its 36 lower 8 x 8 blocks, block (m, k)
// at li_blk(m, k), element (r, q) of it at li_el(r, q): the exclusive or
// spreads the fragment loads of two rows over all bank groups.
constexpr int LT_WP = 66;  // pitch (double2) of a working tile: fragment loads conflict-free
constexpr int LI_N = 36 * 64;
__device__ __forceinline__ int li_blk(int m, int k) { return (m * (m + 1) / 2 + k) * 64; }
__device__ __forceinline__ int li_el(int r, int q) { return r * 8 + (q ^ ((r & 1) << 2)); }
constexpr size_t LP_SMEM_T = (size_t)(LI_N + LDL_NB * LT_WP + LDL_NB) * sizeof(double2);

// Rows of Linv W for this warp's eight columns c0..: accr/acci[m][e] is
// entry (8 m + g, c0 + 2 t4 + e).
__device__ __forceinline__ void lp_linv_product(const double2* __restrict__ Li, const double2* __restrict__ Wt, int c0,
                                                int g, int t4, double (&accr)[8][2], double (&acci)[8][2])
{
#pragma unroll
    for (int m = 0; m < 8; m++)
#pragma unroll
        for (int e = 0; e < 2; e++) accr[m][e] = acci[m][e] = 0.0;
#pragma unroll
    for (int k = 0; k < 8; k++)
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const double2 w = Wt[(8 * k + 4 * h + t4) * LT_WP + c0 + g];
            const double wn = -w.y;
#pragma unroll
            for (int m = k; m < 8; m++) {
                const double2 x = Li[li_blk(m, k) + li_el(g, 4 * h + t4)];
                lp_mma(accr[m][0], accr[m][1], x.x, w.x);
                lp_mma(acci[m][0], acci[m][1], x.x, w.y);
                lp_mma(accr[m][0], accr[m][1], x.y, wn);
                lp_mma(acci[m][0], acci[m][1], x.y, w.x);
            }
        }
}

__device__ void lp_panel(cd* __restrict__ A, int ld, int n, int s, int C, const cd* __restrict__ invD,
                         const cd* __restrict__ linv, double2* sm)
{
    double2* Li = sm;
    double2* Wt = Li + LI_N;                // Wt[q * LT_WP + c]
    double2* ids = Wt + LDL_NB * LT_WP;     // invD of the panel
    const int p0 = s * LDL_NB;              // a panel with columns beyond it is 64 rows high
    const int cb = C * LDL_NB, wd = min(LDL_NB, n - cb);
    const int tid = threadIdx.x, lane = tid & 31, wp = tid >> 5;
    const int g = lane >> 2, t4 = lane & 3;
#pragma unroll 3
    for (int e = tid; e < LI_N; e += 256) {
        const int blk = e >> 6, r = (e >> 3) & 7, q = e & 7;
        const int m = (int)((sqrtf(8.0f * blk + 1.0f) - 1.0f) * 0.5f), k = blk - m * (m + 1) / 2;
        cp_async16(Li + blk * 64 + li_el(r, q), linv + (size_t)(p0 + 8 * m + r) * LDL_NB + 8 * k + q, 16);
    }
#pragma unroll 4
    for (int e = tid; e < LDL_NB * LDL_NB; e += 256) {
        const int q = e & 63, c = e >> 6;
        const bool in = c < wd;
        cp_async16(Wt + q * LT_WP + c, in ? (const void*)(A + (size_t)(p0 + q) + (size_t)(cb + c) * ld) : (const void*)A,
                   in ? 16 : 0);
    }
    cp_async_commit();
    if (tid < LDL_NB) ids[tid] = lp_ldcg(invD + p0 + tid);
    cp_async_wait<0>();
    __syncthreads();
    double accr[8][2], acci[8][2];
    const int c0 = 8 * wp;
    lp_linv_product(Li, Wt, c0, g, t4, accr, acci);
#pragma unroll
    for (int m = 0; m < 8; m++) {
        const double2 d = ids[8 * m + g];
#pragma unroll
        for (int e = 0; e < 2; e++) {
            const int c = c0 + 2 * t4 + e;
            if (c < wd)
                A[(size_t)(p0 + 8 * m + g) + (size_t)(cb + c) * ld] = cmul(cd{accr[m][e], acci[m][e]}, cd{d.x, d.y});
        }
    }
    fence_async_global();  // read by TMA in the updates
    fence_async_shared();  // and this memory is written by TMA next
}

struct alignas(64) LpArgs {
    CUtensorMap t64, t32;   // F's rows 0..n-1 as doubles by columns: boxes of 8 complex rows x 64 and x 32 columns
    cd* A;
    int ld, n, np;
    const unsigned* tasks;  // the list of the CTAs other than the chain CTA
    int ntasks;
    unsigned* cnt;          // tile counters
    unsigned* hc;           // per tile: column halves of band updates finished
    unsigned* cl;           // per tile: panels claimed by a merged update under way
    unsigned* ctl;          // [0] next list index, [1] abort word, [2] trace records, [3] chain CTA's SM + 1
    cd* dw;
    cd* invD;
    cd* linv;               // inverse unit-lower diagonal blocks, row r of panel p at [(64 p + r) * 64]
    int* status;
    const int* limitp;      // poll limit of the bounded waits
    unsigned long long* trace;  // optional: per task (code | cta << 32 | panels << 48, start, ready, done)
};

// B(s, R, C): W(r, c) -= sum_q conj(U(q, r)) d_q U(q, c) over the 64 x 64
// tile, r <= c on a diagonal tile (its diagonal in dw).  Eight warps as
// 2 x 4, each a 32 x 16 complex sub-tile of 8 x 8 mma tiles; the tile's
// old values are the accumulators' initial values (the minus sign is folded
// into the operand -d U(q, c)), so a product is accumulated straight onto
// them.  m consecutive panels s..s+m-1 (whose rows are contiguous) are
// applied in one pass when they are all ready: a rank-64m update, the
// tile read and written once.
// U(s, R) and U(s, C) come by TMA, eight k rows a stage, through a ring of
// TMA_ST stages: thread 0 refills a stage once the eight warps have left it
// (two chunks behind its own), each warp waits only for its data, and no
// barrier stands between chunks.  The 128-byte swizzle puts row k of column
// c at 16-byte slot c * 8 + (k ^ (c & 7)); with the columns of an 8 x 8 mma
// tile taken in the order p(g) = 0 4 1 5 2 6 3 7 a quarter-warp's fragment
// load meets eight different bank groups.  What bounds it: the FP64 tensor
// cores (8.4 us of an SM per panel).  Two CTAs an SM, four panels a pass:
// 17.6 us per panel and pair of CTAs (95 % of the pipe) against 22.0 with
// cp.async stages and two barriers a chunk, whose address arithmetic and
// waits kept the pipe at 68 % (ncu).
// MT x NT mma tiles per warp, WR x WC warps: <4, 2, 2, 4> covers the whole
// 64 x 64 tile, <2, 2, 4, 2> the 64 x 32 column half `half` of it.
template <bool CPLX, int MT, int NT, int WR, int WC>
__device__ bool lp_update(const LpArgs& a, int s, int m, int R, int C, int half, double2* sm, TmaRing& ring)
{
    static_assert(WR * WC == 8 && WR * MT * 8 == LDL_NB, "eight warps over the 64 tile rows");
    constexpr int CW = WC * NT * 8;  // columns covered
    const int tid = threadIdx.x, lane = tid & 31, wp = tid >> 5;
    const int wr = wp / WC, wc = wp % WC;
    const int g = lane >> 2, t4 = lane & 3;
    const int pg = (g & 1) << 2 | g >> 1;
    const int n = a.n, ld = a.ld;
    cd* __restrict__ A = a.A;
    const int p0 = s * LDL_NB;
    const int rb = R * LDL_NB, cb = C * LDL_NB + half * CW;
    const bool dtile = (R == C);
    const unsigned base = (smem32(sm) + 1023u) & ~1023u;
    double2* stages = sm + (base - smem32(sm)) / sizeof(double2);
    double2* dp = stages + TMA_ST * 2 * LP_OP;  // pivots d_q of panels s..s+m-1
    const int nch = m * (LDL_NB / TMA_KC);      // panels with rows below them are whole
    auto issue = [&](int ch, int st) {
        const unsigned bar = ring.full + 8u * st, dst = base + (unsigned)(st * 2 * LP_OP * sizeof(double2));
        bar_expect(bar, (unsigned)((LP_OP + TMA_KC * CW) * sizeof(double2)));
        tma_box(dst, &a.t64, p0 + ch * TMA_KC, rb, bar);
        tma_box(dst + (unsigned)(LP_OP * sizeof(double2)), CW == LDL_NB ? &a.t64 : &a.t32, p0 + ch * TMA_KC, cb, bar);
    };
    // the stage refilled next (thread 0) and the parity its last use ends with
    int rst = ring.st;
    unsigned rph = ring.ph;
    if (tid == 0) {
        fence_async_global();  // the panel rows were written by other CTAs' ordinary stores
        int st = ring.st;
        unsigned ph = ring.ph;
        for (int ch = 0; ch < min(TMA_ST, nch); ch++) {
            issue(ch, st);
            ring.step(st, ph);
        }
    }
    for (int q = tid; q < m * LDL_NB; q += 256) dp[q] = lp_ldcg(a.dw + p0 + q);
    // a warp whose sub-tile lies wholly below the diagonal has nothing to do
    const bool wact = !dtile || (wr * MT * 8 <= half * CW + (wc + 1) * NT * 8 - 1);
    double accr[MT][NT][2], acci[MT][NT][2];
#pragma unroll
    for (int mt = 0; mt < MT; mt++)
#pragma unroll
        for (int nt = 0; nt < NT; nt++)
#pragma unroll
            for (int e = 0; e < 2; e++) {
                const int r = rb + (wr * MT + mt) * 8 + pg;
                const int c = cb + (wc * NT + nt) * 8 + 4 * e + t4;
                double2 o = make_double2(0.0, 0.0);
                if (r < n && c < n && r <= c) {
                    if (r == c) {
                        o = lp_ldcg(a.dw + c);
                        o.y = -o.y;  // dw keeps the conjugate of the upper-triangle value
                    } else {
                        o = lp_ldcg(A + (size_t)r + (size_t)c * ld);
                    }
                }
                accr[mt][nt][e] = o.x;
                acci[mt][nt][e] = o.y;
            }
    __syncthreads();  // dp
    bool ok = true;
    const int f0 = pg * TMA_KC + (t4 ^ pg);  // fragment slots of k = t4 and, with ^ 4, of k = 4 + t4
    int ch = 0;
    for (; ch < nch; ch++) {
        ok = bar_wait(ring.full + 8u * ring.st, ring.ph);
        if (!__all_sync(0xffffffffu, ok)) break;
        if (wact) {
            const double2* Us = stages + ring.st * 2 * LP_OP + (wr * MT) * 64;
            const double2* Vs = stages + ring.st * 2 * LP_OP + LP_OP + (wc * NT) * 64;
#pragma unroll
            for (int j = 0; j < 2; j++) {
                const int f = f0 ^ (4 * j);
                const double2 d = dp[ch * TMA_KC + 4 * j + t4];
                double2 u[MT];
                double vr[NT], vi[NT];
#pragma unroll
                for (int mt = 0; mt < MT; mt++) u[mt] = Us[mt * 64 + f];
#pragma unroll
                for (int nt = 0; nt < NT; nt++) {
                    const double2 v = Vs[nt * 64 + f];
                    // -(d v): the unscaled row, negated
                    vr[nt] = CPLX ? -fma(v.x, d.x, -v.y * d.y) : -v.x * d.x;
                    vi[nt] = CPLX ? -fma(v.x, d.y, v.y * d.x) : -v.y * d.x;
                }
#pragma unroll
                for (int nt = 0; nt < NT; nt++) {
                    const double nr = -vr[nt];
#pragma unroll
                    for (int mt = 0; mt < MT; mt++) {
                        lp_mma(accr[mt][nt][0], accr[mt][nt][1], u[mt].x, vr[nt]);
                        lp_mma(acci[mt][nt][0], acci[mt][nt][1], u[mt].x, vi[nt]);
                    }
#pragma unroll
                    for (int mt = 0; mt < MT; mt++) {
                        lp_mma(accr[mt][nt][0], accr[mt][nt][1], u[mt].y, vi[nt]);
                        lp_mma(acci[mt][nt][0], acci[mt][nt][1], u[mt].y, nr);
                    }
                }
            }
        }
        __syncwarp();
        if (lane == 0) bar_arrive(ring.empty + 8u * ring.st);
        ring.step(ring.st, ring.ph);
        if (tid == 0 && ch >= 2 && ch - 2 + TMA_ST < nch) {
            // (without its stage a chunk is not asked for, and its wait runs out)
            if (bar_wait(ring.empty + 8u * rst, rph)) issue(ch - 2 + TMA_ST, rst);
            ring.step(rst, rph);
        }
    }
    if (__syncthreads_or(ok ? 0 : 1)) {
        if (tid == 0) ring_drain(ring.full, rst, rph, nch - ring_refilled(ch, nch));
        return false;
    }
#pragma unroll
    for (int mt = 0; mt < MT; mt++)
#pragma unroll
        for (int nt = 0; nt < NT; nt++)
#pragma unroll
            for (int e = 0; e < 2; e++) {
                const int r = rb + (wr * MT + mt) * 8 + pg;
                const int c = cb + (wc * NT + nt) * 8 + 4 * e + t4;
                if (r >= n || c >= n || c < r) continue;
                if (c == r)
                    a.dw[c] = cd{accr[mt][nt][e], -acci[mt][nt][e]};
                else
                    A[(size_t)r + (size_t)c * ld] = cd{accr[mt][nt][e], acci[mt][nt][e]};
            }
    return true;
}

__device__ __forceinline__ unsigned long long lp_clock()
{
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// The tile counts a list task waits for: cnt[ix[i]] >= need[i], i < the
// returned count.
__device__ __forceinline__ int lp_deps(unsigned task, long long (&ix)[3], unsigned (&need)[3])
{
    const unsigned type = task >> 30;
    const int s = (task >> 20) & 511, R = (task >> 10) & 1023, C = task & 1023;
    ix[1] = ix[2] = 0;
    need[1] = need[2] = 0u;
    if (type == LP_T) {
        ix[0] = lp_tix(s, s), need[0] = (unsigned)s + 1;
        ix[1] = lp_tix(s, C), need[1] = (unsigned)s;
        return 2;
    }
    const int last = lp_grouped(s, R) ? s + LP_MERGE - 1 : s;
    ix[0] = lp_tix(R, C), need[0] = (unsigned)s;
    ix[1] = lp_tix(last, R), need[1] = (unsigned)last + 1;
    ix[2] = lp_tix(last, C), need[2] = (unsigned)last + 1;
    return (R == C) ? 2 : 3;
}

// Thread 0: wait until cnt[ix[i]] >= need[i] for the k (<= 3) conditions,
// polling them together: 1 when they hold, 0 when this CTA must stop.  For
// an update by panel need[0] also 2, as soon as a merged update that covers
// this panel is under way in another CTA: waiting for it to finish, only to
// find the panel applied, held CTAs for 13 % of the run at K = 4000.
__device__ __forceinline__ int lp_wait_all(const LpArgs& a, const long long (&ix)[3], const unsigned (&need)[3],
                                           int k, int limit, bool update = false)
{
    int spins = 0;
    for (;;) {
        if (update && *((volatile unsigned*)(a.cl + ix[0])) > need[0]) return 2;
        unsigned v[3];
#pragma unroll
        for (int i = 0; i < 3; i++) v[i] = (i < k) ? lp_ld_acquire(a.cnt + ix[i]) : 0u;
        bool ok = true;
#pragma unroll
        for (int i = 0; i < 3; i++) ok = ok && (i >= k || v[i] >= need[i]);
        if (ok) return 1;
        if (++spins > limit || *((volatile unsigned*)(a.ctl + 1)) != 0u) {
            atomicExch(a.status + ST_SOLVE_TIMEOUT, 1);
            atomicExch(a.ctl + 1, 1u);
            return 0;
        }
        __nanosleep(32);
    }
}

__device__ __forceinline__ void lp_trace(const LpArgs& a, unsigned code, int m, unsigned long long t0,
                                         unsigned long long t1)
{
    if (!a.trace) return;
    const unsigned long long t2 = lp_clock();
    const unsigned i = atomicAdd(a.ctl + 2, 1u);
    unsigned long long* r = a.trace + 4 * (size_t)i;
    r[0] = (unsigned long long)code | (unsigned long long)blockIdx.x << 32 | (unsigned long long)m << 48;
    r[1] = t0;
    r[2] = t1;
    r[3] = t2;
}

// One task, all threads.  Thread 0 has checked the dependencies; on return
// the task's stores are done (a barrier follows).  m: panels of an update.
// False when a copy did not arrive.
template <bool CPLX>
__device__ __forceinline__ bool lp_exec(const LpArgs& a, unsigned type, int s, int m, int R, int C, int half,
                                        double2* sm, TmaRing& ring)
{
    if (type == LP_T) {
        lp_panel(a.A, a.ld, a.n, s, C, a.invD, a.linv, sm);
        return true;
    }
    if (!lp_grouped(s, R) && lp_split(s, R, C)) return lp_update<CPLX, 2, 2, 4, 2>(a, s, 1, R, C, half, sm, ring);
    return lp_update<CPLX, 4, 2, 2, 4>(a, s, m, R, C, 0, sm, ring);
}

// After the task's barrier: thread 0 publishes the tile's new count.  The
// barrier orders every thread's stores before the gpu-scope release.
__device__ __forceinline__ void lp_publish(const LpArgs& a, long long ix, unsigned v)
{
    if (threadIdx.x == 0) lp_st_release(a.cnt + ix, v);
}

// ---------------------------------------------------------------------------
// The chain CTA: per panel s the three tasks the next diagonal tile waits
// for.
//   D(s)          elimination of [tile | identity], so that L_ss^-1 comes
//                 with U_ss.  Each warp keeps one column of 8 x 8 tiles in
//                 registers: the rows up to its own diagonal tile are W, the
//                 ones below it the identity's column (zero at first), so
//                 every warp always holds eight.  They are held transposed
//                 (lane (g, t4): column g, rows 2 t4 and 2 t4 + 1 of a tile)
//                 because a product's result is then the next product's
//                 first operand without a move.  Per row tile b: the warp of
//                 column b eliminates the 8 x 8 block with the identity
//                 beside it (X_b = L_bb^-1); the others take Y_b = X_b W_b,
//                 write U = invD Y_b or the row of L_ss^-1 out, and share U
//                 through shared memory; then every warp updates its tiles
//                 below with conj(U(b, a))^T Y_b, the warp of column b + 1
//                 only its diagonal tile, which it eliminates beside the
//                 others' products.  Two barriers a row tile.  Published at
//                 once, so the other panel rows start;
//   T(s, s+1)     the tile to its right, as lp_panel does it, kept in shared
//                 memory;
//   B(s, s+1, s+1) the old values of tile (s+1, s+1) once the other CTAs
//                 have applied panels 0..s-1, then panel s, straight into
//                 the registers step s+1 starts from.
// The tile (s+1, s+2) that T(s+1, s+2) needs comes from the other CTAs
// (T(s, s+2), then B(s, s+1, s+2)) while this CTA runs D(s+1).
constexpr int LC_UP = 57;  // pitch of the shared rows of U (columns 8..63): 1 mod 4, conflict-free
constexpr int LC_XP = 9;   // pitch of X_b
constexpr size_t LP_SMEM_C = (size_t)(LI_N + LDL_NB * LT_WP + 2 * LDL_NB + 8 * LC_UP + 8 * LC_XP) * sizeof(double2);
constexpr size_t lp_max(size_t a, size_t b) { return a > b ? a : b; }
constexpr size_t LP_SMEM_BAR = lp_max(LP_SMEM_B, lp_max(LP_SMEM_C, LP_SMEM_T));  // the ring's mbarriers
constexpr size_t LP_SMEM = LP_SMEM_BAR + 2 * TMA_ST * 8;

// 1/d of a normal d, without a branch: the hardware's seed y and the
// geometric series of 1 / (1 - e), e = 1 - d y, to e^2 (|e| is at most
// 2^-19.9 over all upper words of the mantissa, measured: a remainder below
// 2^-59), which rounds once.  It stands in a chain of 64 a tile: the
// 8 x 8 elimination measures 862 cycles with it and 1428 with a reciprocal
// that also covers what lies outside the normal range.
__device__ __forceinline__ double lp_rcp(double d)
{
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(d));
    const double e = fma(-d, y, 1.0);
    return fma(y, fma(e, e, e), y);
}

template <bool CPLX>
__device__ void lp_chain(const LpArgs& a, double2* sm, int limit)
{
    double2* Li = sm;                     // L_ss^-1 by 8 x 8 blocks, for T
    double2* Rt = sm + LI_N;              // right tile, Rt[q * LT_WP + c]
    // pivots d of the panel: real ones in two buffers, so that the next
    // panel's first block can be eliminated while B still reads them
    double2* dpv = Rt + LDL_NB * LT_WP;
    double* dpr = reinterpret_cast<double*>(dpv);
    double2* sinv = dpv + LDL_NB;         // their inverses (invD)
    double2* Us = sinv + LDL_NB;          // -conj(U(b, c)), c >= 8: Us[(row of tile b) * LC_UP + c - 8]
    double2* Xs = Us + 8 * LC_UP;         // X_b(i, j) at Xs[i * LC_XP + j]
    __shared__ int s_go, s_v, s_pre;
    const int tid = threadIdx.x, lane = tid & 31, wp = tid >> 5;
    const int g = lane >> 2, t4 = lane & 3;
    // the column of tiles this warp holds: 9 tiles of B for each pair of
    // warps that shares a scheduler
    const int cw = wp < 4 ? wp : 11 - wp;
    const int n = a.n, ld = a.ld;
    cd* A = a.A;
    auto times = [](cd v, cd r) { return CPLX ? cmul(v, r) : cd{v.x * r.x, v.y * r.x}; };
    double wr[8][2], wi[8][2];  // row tile b + i of the column: rows 2 t4 + e, column g
    double yr[2], yi[2];        // Y_b of the column, the same way
    bool apply = false;         // panel s - 1 is still to be applied to tile (s, s)
    for (int s = 0; s < a.np; s++) {
        const int p0 = s * LDL_NB, b = min(LDL_NB, n - p0);
        const bool right = s + 1 < a.np;
        const int cb = p0 + LDL_NB, wd = right ? min(LDL_NB, n - cb) : 0;
        unsigned long long t0 = 0;
        if (tid == 0 && a.trace) t0 = lp_clock();
        // ================= the rest of B(s-1, s, s)
        // the tile's values from global memory, the whole of the diagonal
        // 8 x 8 tile, the identity beyond the last row, zeros below
        {
            const int c = 8 * cw + g;
            const bool cin = c < b;
            const cd* col = A + (size_t)(p0 + 2 * t4) + (size_t)(p0 + c) * ld;
#pragma unroll
            for (int i = 0; i < 8; i++)
#pragma unroll
                for (int e = 0; e < 2; e++) {
                    double2 w = make_double2(0.0, 0.0);
                    if (i < cw && cin) w = lp_ldcg(col + 8 * i + e);
                    wr[i][e] = w.x;
                    wi[i][e] = w.y;
                }
#pragma unroll
            for (int e = 0; e < 2; e++) {
                const int r = 8 * cw + 2 * t4 + e;
                double2 w = make_double2((r == c) ? 1.0 : 0.0, 0.0);
                if (max(r, c) < b) {
                    w = lp_ldcg(r == c ? a.dw + p0 + r : A + (size_t)(p0 + min(r, c)) + (size_t)(p0 + max(r, c)) * ld);
                    if (r >= c) w.y = -w.y;  // dw keeps the conjugate of the upper-triangle value
                }
#pragma unroll
                for (int i = 0; i < 8; i++)
                    if (i == cw) {
                        wr[i][e] = w.x;
                        wi[i][e] = w.y;
                    }
            }
        }
        if (apply) {
            // W(a, cw)^T -= (d U(:, cw))^T conj(U(:, a)); columns beyond the
            // last row are zero in the right tile
#pragma unroll 1
            for (int k0 = 0; k0 < LDL_NB; k0 += 8) {
                const double2* row = Rt + (k0 + t4) * LT_WP + g;
                double vr[2], vi[2];
#pragma unroll
                for (int k = 0; k < 2; k++) {
                    const double2 uc = row[4 * k * LT_WP + 8 * cw];
                    const int q = k0 + 4 * k + t4;
                    const double2 d = CPLX ? dpv[q] : make_double2(dpr[((s - 1) & 1) * LDL_NB + q], 0.0);
                    vr[k] = CPLX ? -fma(uc.x, d.x, -uc.y * d.y) : -uc.x * d.x;
                    vi[k] = CPLX ? -fma(uc.x, d.y, uc.y * d.x) : -uc.y * d.x;
                }
#pragma unroll
                for (int i = 0; i < 8; i++)
                    if (i <= cw) {
#pragma unroll
                        for (int k = 0; k < 2; k++) {
                            const double2 u = row[4 * k * LT_WP + 8 * i];
                            lp_mma(wr[i][0], wr[i][1], vr[k], u.x);
                            lp_mma(wi[i][0], wi[i][1], vi[k], u.x);
                            lp_mma(wr[i][0], wr[i][1], vi[k], u.y);
                            lp_mma(wi[i][0], wi[i][1], vr[k], -u.y);
                        }
                    }
            }
        }
        if (CPLX) __syncthreads();  // one buffer of pivots
        if (tid == 0 && s > 0) {
            lp_trace(a, lp_code(LP_B, s - 1, s, s), apply ? 1 : 0, t0, t0);
            if (a.trace) t0 = lp_clock();
        }
        // ================= D(s)
        // bk = -1: the first diagonal tile alone; then per row tile (one
        // call site of the elimination keeps the code small)
        // this warp's eight columns of the right tile
        auto load_right = [&]() {
#pragma unroll 4
            for (int e = lane; e < 8 * LDL_NB; e += 32) {
                const int q = e & 63, c = 8 * wp + (e >> 6);
                const bool in = c < wd;
                cp_async16(Rt + q * LT_WP + c,
                           in ? (const void*)(A + (size_t)(p0 + q) + (size_t)(cb + c) * ld) : (const void*)A, in ? 16 : 0);
            }
            cp_async_commit();
        };
        // is tile (s, s+1) ready already?  Then its columns are fetched during D
        if (tid == 128) s_pre = right && lp_ld_acquire(a.cnt + lp_tix(s, s + (right ? 1 : 0))) >= (unsigned)s;
#pragma unroll 1
        for (int bk = -1; bk < 8; bk++) {
            if (bk < 0) {
                // L_ss^-1 is zero above its diagonal blocks
                cd* z = a.linv + (size_t)(p0 + (lane >> 3)) * LDL_NB + 8 * cw + (lane & 7);
                for (int r = lane >> 3; r < min(8 * cw, b); r += 4, z += 4 * LDL_NB) *z = cd{0.0, 0.0};
            }
            // each warp at a step at which no other waits for it
            if (bk == ((cw + 4) & 7) && s_pre) load_right();
            if (bk >= 0) {
                if (cw != bk) {
                    double zr[2][2], zi[2][2];  // the two halves of the sum, chains of two products each
#pragma unroll
                    for (int e = 0; e < 2; e++) {
                        const double2 x = Xs[g * LC_XP + 2 * t4 + e];
                        zr[e][0] = zr[e][1] = zi[e][0] = zi[e][1] = 0.0;
                        lp_mma(zr[e][0], zr[e][1], wr[0][e], x.x);
                        lp_mma(zi[e][0], zi[e][1], wr[0][e], x.y);
                        lp_mma(zr[e][0], zr[e][1], -wi[0][e], x.y);
                        lp_mma(zi[e][0], zi[e][1], wi[0][e], x.x);
                    }
#pragma unroll
                    for (int e = 0; e < 2; e++) {
                        yr[e] = zr[0][e] + zr[1][e];
                        yi[e] = zi[0][e] + zi[1][e];
                    }
                    if (cw > bk) {
#pragma unroll
                        for (int e = 0; e < 2; e++) {
                            const double2 id = sinv[8 * bk + 2 * t4 + e];
                            const cd u = times(cd{yr[e], yi[e]}, cd{id.x, id.y});
                            Us[(2 * t4 + e) * LC_UP + 8 * cw + g - 8] = make_double2(-u.x, u.y);
                            if (8 * cw + g < b)
                                A[(size_t)(p0 + 8 * bk + 2 * t4 + e) + (size_t)(p0 + 8 * cw + g) * ld] = u;
                        }
                    }
                } else {
                    // what the elimination of this block left, written out
                    // while the other warps multiply
                    const double2* ub = Li + li_blk(7, 7);
#pragma unroll
                    for (int h = 0; h < 2; h++) {
                        const int i = (lane >> 3) + 4 * h, j = lane & 7, r = 8 * bk + i;
                        const double2 v = Xs[i * LC_XP + j], u = ub[8 * i + j];
                        if (bk < 7) Li[li_blk(bk, bk) + li_el(i, j)] = v;
                        if (r < b) {
                            cd* row = a.linv + (size_t)(p0 + r) * LDL_NB + 8 * bk + j;
                            *row = cd{v.x, v.y};
                            if (i < j && 8 * bk + j < b) A[(size_t)(p0 + r) + (size_t)(p0 + 8 * bk + j) * ld] = cd{u.x, u.y};
                        }
                    }
                    if (lane < 8 && 8 * bk + lane < b) {
                        const int r = 8 * bk + lane;
                        const double2 id = sinv[r], d = CPLX ? dpv[r] : make_double2(dpr[(s & 1) * LDL_NB + r], 0.0);
                        a.invD[p0 + r] = cd{id.x, id.y};
                        a.dw[p0 + r] = cd{d.x, d.y};
                        if (d.x == 0.0 && d.y == 0.0) atomicCAS(a.status + ST_ZERO_PIVOT, 0, p0 + r + 1);
                    }
                }
                __syncthreads();
                if (bk == 7 && cw == 7) {  // its own block last: it kept U(7, 7)'s place
#pragma unroll
                    for (int h = 0; h < 2; h++) {
                        const int i = (lane >> 3) + 4 * h, j = lane & 7;
                        Li[li_blk(7, 7) + li_el(i, j)] = Xs[i * LC_XP + j];
                    }
                }
                if (cw < bk) {
#pragma unroll
                    for (int e = 0; e < 2; e++) {
                        const int rr = 2 * t4 + e;
                        Li[li_blk(bk, cw) + li_el(rr, g)] = make_double2(yr[e], yi[e]);
                        if (8 * bk + rr < b)
                            a.linv[(size_t)(p0 + 8 * bk + rr) * LDL_NB + 8 * cw + g] = cd{yr[e], yi[e]};
                    }
                }
                if (bk < 7) {
                    // W(a, cw) -= conj(U(b, a))^T Y_b, the tiles moving up one place
                    const int lim = cw > bk ? cw - bk : 7 - bk;
                    const double2* u0 = Us + 2 * t4 * LC_UP + 8 * bk - 8 + g;
#pragma unroll
                    for (int i = 1; i < 8; i++) {
                        if (i <= lim) {
#pragma unroll
                            for (int e = 0; e < 2; e++) {
                                const double2 v = u0[e * LC_UP + 8 * i];
                                lp_mma(wr[i][0], wr[i][1], yr[e], v.x);
                                lp_mma(wi[i][0], wi[i][1], yi[e], v.x);
                                lp_mma(wr[i][0], wr[i][1], yi[e], -v.y);
                                lp_mma(wi[i][0], wi[i][1], yr[e], v.y);
                            }
                        }
#pragma unroll
                        for (int e = 0; e < 2; e++) {
                            wr[i - 1][e] = wr[i][e];
                            wi[i - 1][e] = wi[i][e];
                        }
                    }
                }
            }
            if (cw == bk + 1) {
                // eliminate the 8 x 8 block with the identity beside it: lane
                // (hf, c) holds the rows 2 k + hf of column c (0..7 the
                // block's, 8..15 the identity's), the pivot row goes round
                // through Xs; row i takes conj(W(q, i)) W(q, :) / d, whose
                // product does not wait for the reciprocal
                const int c = lane & 15, hf = lane >> 4;
                const bool col = c < 8;
#pragma unroll
                for (int e = 0; e < 2; e++) Xs[(2 * t4 + e) * LC_XP + g] = make_double2(wr[0][e], wi[0][e]);
                __syncwarp();
                cd x[4];
#pragma unroll
                for (int k = 0; k < 4; k++) {
                    double2 v = make_double2((2 * k + hf + 8 == c) ? 1.0 : 0.0, 0.0);
                    if (col) v = Xs[(2 * k + hf) * LC_XP + c];
                    x[k] = cd{v.x, v.y};
                }
#pragma unroll
                for (int q = 0; q < 8; q++) {
                    const int kq = q >> 1, hq = q & 1;
                    const cd d = lp_shfl(x[kq], q + 16 * hq), xq = lp_shfl(x[kq], c + 16 * hq);
                    if (q > 0) {
                        __syncwarp();
                        if (col && hf == hq) Xs[q * LC_XP + c] = make_double2(x[kq].x, x[kq].y);
                        __syncwarp();
                    }
                    cd id;
                    if (CPLX) {
                        const double r = __drcp_rn(fma(d.x, d.x, d.y * d.y));
                        id = cd{d.x * r, -d.y * r};
                    } else {
                        id = cd{lp_rcp(d.x), 0.0};
                    }
#pragma unroll
                    for (int k = kq; k < 4; k++) {
                        const double2 w = Xs[q * LC_XP + 2 * k + hf];
                        const cd t = cmul(cd{w.x, -w.y}, xq);
                        const cd v = CPLX ? cfms(conj(id), t, x[k]) : cd{fma(-id.x, t.x, x[k].x), fma(-id.x, t.y, x[k].y)};
                        if (k > kq || hf > hq) x[k] = v;
                    }
                    if (col && hf == hq) x[kq] = times(x[kq], id);  // U(q, c)
                    if (lane == q + 16 * hq) {
                        // an exactly zero pivot is reported; its 1/d stays 0
                        const bool zero = d.x == 0.0 && (!CPLX || d.y == 0.0);
                        if (CPLX)
                            dpv[8 * cw + q] = make_double2(d.x, d.y);
                        else
                            dpr[(s & 1) * LDL_NB + 8 * cw + q] = d.x;
                        sinv[8 * cw + q] = make_double2(zero ? 0.0 : id.x, zero ? 0.0 : id.y);
                    }
                }
                __syncwarp();
                {
                    // X_b to its place; U(b, b) waits where the last block of
                    // L_ss^-1 goes
                    double2* out = col ? Li + li_blk(7, 7) + 8 * hf + c : Xs + hf * LC_XP + c - 8;
                    const int step = col ? 16 : 2 * LC_XP;
#pragma unroll
                    for (int k = 0; k < 4; k++) out[k * step] = make_double2(x[k].x, x[k].y);
                }
                __syncwarp();
#pragma unroll
                for (int e = 0; e < 2; e++) {
                    const double2 v = Xs[(2 * t4 + e) * LC_XP + g];
                    yr[e] = v.x;
                    yi[e] = v.y;
                }
                // the column turns into the identity's: nothing below it yet
#pragma unroll
                for (int i = 0; i < 8; i++) wr[i][0] = wr[i][1] = wi[i][0] = wi[i][1] = 0.0;
            }
            __syncthreads();
        }
        lp_publish(a, lp_tix(s, s), (unsigned)s + 1);
        if (tid == 0) lp_trace(a, lp_code(LP_D, s, s, s), 1, t0, t0);
        if (!right) break;
        // ================= T(s, s+1)
        if (tid == 0) {
            if (a.trace) t0 = lp_clock();
            s_go = 1;
            long long ix[3] = {lp_tix(s, s + 1), 0, 0};
            unsigned need[3] = {(unsigned)s, 0u, 0u};
            if (!s_pre) s_go = lp_wait_all(a, ix, need, 1, limit);
        }
        __syncthreads();
        if (!s_go) return;
        unsigned long long t1 = 0;
        if (tid == 0 && a.trace) t1 = lp_clock();
        if (!s_pre) load_right();
        cp_async_wait<0>();
        __syncwarp();  // a warp multiplies the columns it has loaded
        {
            // each warp reads and rewrites its own eight columns of the right tile
            const int c0 = 8 * wp;
            lp_linv_product(Li, Rt, c0, g, t4, wr, wi);
            __syncwarp();
#pragma unroll
            for (int m = 0; m < 8; m++) {
                const double2 d = sinv[8 * m + g];
#pragma unroll
                for (int e = 0; e < 2; e++) {
                    const int c = c0 + 2 * t4 + e;
                    const cd u = times(cd{wr[m][e], wi[m][e]}, cd{d.x, d.y});
                    Rt[(8 * m + g) * LT_WP + c] = make_double2(u.x, u.y);
                    if (c < wd) A[(size_t)(p0 + 8 * m + g) + (size_t)(cb + c) * ld] = u;
                }
            }
        }
        fence_async_global();
        __syncthreads();
        lp_publish(a, lp_tix(s, s + 1), (unsigned)s + 1);
        if (tid == 0) lp_trace(a, lp_code(LP_T, s, s, s + 1), 1, t0, t1);
        // ================= B(s, s+1, s+1): the wait; the products follow at
        // the top of the next step
        if (tid == 0) {
            long long ix[3] = {lp_tix(s + 1, s + 1), 0, 0};
            unsigned need[3] = {(unsigned)s, 0u, 0u};
            const int go = lp_wait_all(a, ix, need, 1, limit);
            s_go = go;
            s_v = go ? (int)lp_ld_acquire(a.cnt + ix[0]) : 0;
        }
        __syncthreads();
        if (!s_go) return;
        apply = s_v == s;  // panels already applied to tile (s+1, s+1)
    }
}

// CTA 0 runs the critical chain, per panel s: D(s), then T(s, s+1) and
// B(s, s+1, s+1), which D(s+1) needs; D(s) is published before the other
// two so that the panel rows of the other tiles start at once.  The other
// CTAs take every remaining task from the list, each when it is free.  An update B(s, R, C)
// whose tile already carries more than s panels (applied by an earlier
// merged update) does nothing; otherwise it also applies the following
// panels s+1.. (up to LP_MERGE in all, below R) whose panel rows of R and
// C are already final.
template <bool CPLX>
__global__ void __launch_bounds__(256, 2) k_ldl_persist(const __grid_constant__ LpArgs a)
{
    extern __shared__ double2 lsm[];
    __shared__ unsigned s_next;
    __shared__ int s_go, s_m;
    const int tid = threadIdx.x;
    const int limit = *((const volatile int*)a.limitp);
    // the chain CTA has its SM to itself: it publishes its SM, and the CTA
    // sharing that SM takes no tasks
    if (tid == 0) {
        unsigned smid;
        asm volatile("mov.u32 %0, %%smid;" : "=r"(smid));
        int go = 1;
        if (blockIdx.x == 0) {
            lp_st_release(a.ctl + 3, smid + 1);
        } else {
            int spins = 0;
            unsigned v;
            while ((v = lp_ld_acquire(a.ctl + 3)) == 0u) {
                if (++spins > limit || *((volatile unsigned*)(a.ctl + 1)) != 0u) {
                    atomicExch(a.status + ST_SOLVE_TIMEOUT, 1);
                    atomicExch(a.ctl + 1, 1u);
                    break;
                }
                __nanosleep(32);
            }
            go = (v != 0u && v != smid + 1);
        }
        s_go = go;
    }
    __syncthreads();
    if (!s_go) return;
    if (blockIdx.x == 0) {
        lp_chain<CPLX>(a, lsm, limit);
        return;
    }
    TmaRing ring;
    ring.init(smem32(lsm) + (unsigned)LP_SMEM_BAR, tid);
    __syncthreads();
    for (;;) {
        unsigned long long t0 = 0, t1 = 0;
        if (tid == 0) {
            if (a.trace) t0 = lp_clock();
            // the next task in list order, taken when this CTA is free (a
            // task fetched earlier could wait behind a long update)
            unsigned task = LP_NONE;
            if (*((volatile unsigned*)(a.ctl + 1)) == 0u) {
                const unsigned i = atomicAdd(a.ctl, 1u);
                if (i < (unsigned)a.ntasks) task = __ldg(a.tasks + i);
            }
            int go = 0, m = 1;
            if (task != LP_NONE) {
                const unsigned type = task >> 30;
                const int s = (task >> 20) & 511, R = (task >> 10) & 1023, C = task & 1023;
                long long ix[3] = {0, 0, 0};
                unsigned need[3] = {0u, 0u, 0u};
                const int k = lp_deps(task, ix, need);
                const bool group = type == LP_B && lp_grouped(s, R);
                const bool whole = type == LP_B && !group && !lp_split(s, R, C);
                if (group) m = LP_MERGE;
                go = lp_wait_all(a, ix, need, k, limit, whole);
                if (go == 1 && type == LP_B && !group) {
                    if (lp_ld_acquire(a.cnt + ix[0]) > (unsigned)s) {
                        go = 2;  // applied already by a merged update
                    } else if (whole) {
                        // following panels whose rows of R and C are final
                        unsigned fr[LP_MERGE - 1], fc[LP_MERGE - 1];
#pragma unroll
                        for (int j = 1; j < LP_MERGE; j++) {
                            const bool in = s % LP_MERGE + j < LP_MERGE && s + j < R;
                            fr[j - 1] = in ? lp_ld_acquire(a.cnt + lp_tix(s + j, R)) : 0u;
                            fc[j - 1] = (in && R != C) ? lp_ld_acquire(a.cnt + lp_tix(s + j, C)) : 0u;
                        }
#pragma unroll
                        for (int j = 1; j < LP_MERGE; j++) {
                            const unsigned want = (unsigned)(s + j) + 1;
                            // the panels of the band next to row R (split in column
                            // halves) and the chain's own update keep their own short
                            // tasks: a long merged update would hold up the panel rows
                            // the chain waits for
                            const bool own = lp_split(s + j, R, C) || (s + j == R - 1);
                            if (m == j && !own && s % LP_MERGE + j < LP_MERGE && s + j < R && fr[j - 1] >= want && (R == C || fc[j - 1] >= want))
                                m = j + 1;
                        }
                        if (m > 1) *((volatile unsigned*)(a.cl + ix[0])) = (unsigned)(s + m);
                    }
                }
                if (!go) task = LP_NONE;
            }
            s_next = task;
            s_go = go;
            s_m = m;
            if (a.trace) t1 = lp_clock();
        }
        __syncthreads();
        const unsigned task = s_next;
        const int go = s_go, m = s_m;
        if (task == LP_NONE) return;
        const unsigned type = task >> 30;
        const int s = (task >> 20) & 511, R = (task >> 10) & 1023, C = task & 1023;
        const int half = (task >> 29) & 1;
        if (go == 1) {
            if (!lp_exec<CPLX>(a, type, s, m, R, C, half, lsm, ring)) {
                // a copy did not arrive, and none is in flight: report, stop
                if (tid == 0) {
                    atomicExch(a.status + ST_SOLVE_TIMEOUT, 1);
                    atomicExch(a.ctl + 1, 1u);
                }
                return;
            }
            __syncthreads();
            const long long tt = (type == LP_B) ? lp_tix(R, C) : lp_tix(s, (type == LP_D) ? s : C);
            if (type == LP_B && !lp_grouped(s, R) && lp_split(s, R, C)) {
                // a column half: the second of the two to finish publishes the tile
                if (tid == 0) {
                    unsigned old;
                    asm volatile("atom.acq_rel.gpu.global.add.u32 %0, [%1], 1;" : "=r"(old) : "l"(a.hc + tt) : "memory");
                    if (old & 1u) lp_st_release(a.cnt + tt, (unsigned)s + 1);
                }
            } else {
                lp_publish(a, tt, (unsigned)(s + m));
            }
        }
        if (tid == 0) lp_trace(a, task, go == 1 ? m : 0, t0, t1);
        __syncthreads();  // s_next, s_go, s_m are rewritten by the next task
    }
}

// Grid of the persistent kernel (co-resident CTAs), 0 if unavailable.
int ldlp_grid(Ctx& c)
{
    if (!c.attr_lp) {
        if (cudaFuncSetAttribute(k_ldl_persist<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)LP_SMEM) !=
                cudaSuccess ||
            cudaFuncSetAttribute(k_ldl_persist<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)LP_SMEM) !=
                cudaSuccess) {
            cudaGetLastError();
            return 0;
        }
        c.attr_lp = true;
    }
    if (c.lp_grid > 0) return c.lp_grid;
    int per_sm = 0, sms = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_ldl_persist<false>, 256, LP_SMEM) != cudaSuccess ||
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, c.dev) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    int coop = 0;
    cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, c.dev);
    if (!coop || per_sm < 1) return 0;
    c.lp_grid = per_sm * sms;
    c.lp_sms = sms;
    return c.lp_grid;
}

// The task list of an n-row factorisation in device memory (owned by the
// caller, freed with cudaFree; at least one entry); *count receives its
// length (0 when the chain CTA does everything).
int ldlp_tasks(Ctx& c, int n, unsigned** tasks, int* count)
{
    const int grid = ldlp_grid(c);
    if (grid <= 0) return -1;
    const int np = (n + LDL_NB - 1) / LDL_NB;
    if (n > LDL_PERSIST_MAX) return -1;
    const int per_sm = std::max(1, c.lp_grid / std::max(1, c.lp_sms));
    std::vector<unsigned> list;
    lp_schedule(np, std::max(1, grid - per_sm), LpCost(), true, list);
    unsigned* d = nullptr;
    if (cudaMalloc(&d, std::max<size_t>(1, list.size()) * sizeof(unsigned)) != cudaSuccess) {
        cudaGetLastError();
        return -3;
    }
    if (!list.empty() &&
        cudaMemcpy(d, list.data(), list.size() * sizeof(unsigned), cudaMemcpyHostToDevice) != cudaSuccess) {
        cudaFree(d);
        return -2;
    }
    *tasks = d;
    *count = (int)list.size();
    return 0;
}

// Number of tasks of an n-row factorisation, the chain's included.
long long ldlp_task_total(int n)
{
    const long long np = (n + LDL_NB - 1) / LDL_NB;
    long long split = 0;  // the second column halves of the band updates
    for (long long s = 0; s + 2 < np; s++) split += 2 * (np - s - 2);
    return np + np * (np - 1) / 2 + (np - 1) * np * (np + 1) / 6 + split;
}

// Tile counters and the control words (next task, abort word, trace
// records, the chain CTA's SM), once for the largest factorisation this
// context can take here (60 KB at 5000 rows, 0.24 MB at 12800).  The cached
// graphs of every size hold this address, so it never moves.
int ldlp_reserve(Ctx& c)
{
    if (c.lp_cnt) return 0;
    const size_t np = (std::min(c.ld, LDL_PERSIST_MAX) + LDL_NB - 1) / LDL_NB;
    if (cudaMalloc(&c.lp_cnt, (np * (np + 1) / 2 * 3 + 4) * sizeof(unsigned)) != cudaSuccess) {
        cudaGetLastError();
        c.lp_cnt = nullptr;
        return -3;
    }
    return 0;
}

// Queue one persistent factorisation of rows 0..n-1 (the working upper
// triangle and dw already initialised by k_ldl_mirror); trace (device,
// 4 x ldlp_task_total(n) values) may be null.
int ldlp_enqueue(Ctx& c, int n, const unsigned* tasks, int ntasks, unsigned long long* trace)
{
    const int np = (n + LDL_NB - 1) / LDL_NB;
    const size_t ntile = (size_t)np * (np + 1) / 2;
    cudaMemsetAsync(c.lp_cnt, 0, (3 * ntile + 4) * sizeof(unsigned), c.stream);
    LpArgs a;
    if (!tma_map(&a.t64, c.F, c.ld, n, n, LDL_NB) || !tma_map(&a.t32, c.F, c.ld, n, n, LDL_NB / 2)) return -2;
    a.A = c.F;
    a.ld = c.ld;
    a.n = n;
    a.np = np;
    a.tasks = tasks;
    a.ntasks = ntasks;
    a.cnt = c.lp_cnt;
    a.hc = c.lp_cnt + ntile;
    a.ctl = c.lp_cnt + 2 * ntile;
    a.cl = c.lp_cnt + 2 * ntile + 4;
    a.dw = c.dw;
    a.invD = c.invD;
    a.linv = c.linv;
    a.status = c.status;
    a.limitp = c.counters + 3;
    a.trace = trace;
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.gridDim = dim3(std::min(c.lp_grid, 1 + ntasks));
    cfg.blockDim = dim3(256);
    cfg.dynamicSmemBytes = LP_SMEM;
    cfg.stream = c.stream;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    if (c.pivot_mode)
        cudaLaunchKernelEx(&cfg, k_ldl_persist<true>, a);
    else
        cudaLaunchKernelEx(&cfg, k_ldl_persist<false>, a);
    c.launches++;
    return 0;
}

}  // namespace ecg

// Host-only diagnostics: the tasks of the persistent factorisation of n rows
// for a grid of `workers` CTAs in the scheduler's start order, the chain
// CTA's included.  No GPU needed.
static int task_order(int n, int workers, bool group, unsigned* out, long long cap, long long* count)
{
    using namespace ecg;
    if (n < 1 || workers < 1 || !count) return -1;
    const int np = (n + LDL_NB - 1) / LDL_NB;
    if (np > 200) return -1;
    std::vector<unsigned> full, list;
    lp_schedule(np, workers, LpCost(), group, list, &full);
    *count = (long long)full.size();
    if (out && cap >= (long long)full.size()) std::copy(full.begin(), full.end(), out);
    return 0;
}

// Every update a task of its own, which the kernel does not run.
extern "C" int ecg_ldl_schedule(int n, int workers, unsigned* out, long long cap, long long* count)
{
    return task_order(n, workers, false, out, cap, count);
}

// What the kernel runs: its list is this order without the chain's tasks.
extern "C" int ecg_ldl_task_list(int n, int workers, unsigned* out, long long cap, long long* count)
{
    return task_order(n, workers, true, out, cap, count);
}
