// k_chol_dag.cu -- FP64 tile Cholesky as ONE persistent launch that walks the
// task DAG on the device.
//
// Reference: dchol_rl (chol_rlmain.c:22-53) issues POTRF / TRSM / SYRK / GEMM
// tile tasks that the OmpSs runtime orders by their data dependencies (keyed
// on tile base addresses, tasks_potrf.h:19) and by priority (POTRF and TRSM
// at 9999 over GEMM and SYRK at 9, chol_rlmain.c:14-19).  Here the DAG lives
// on the GPU:
//
//   * The factor is cut into 64 x 64 tiles (the last row and column ragged).
//     Three kinds of tasks, all left-looking:
//       T(i, j), i >= j + 2:  S = A_ij - sum_{k<j} L_ik L_jk^T,  L_ij = S W_j^T
//       P(j), j >= 3:  A_{j,j-1} -= sum_{k<j-2} L_jk L_{j-1,k}^T, in place
//       M(j):  S = A_jj - sum_{k<j-1} L_jk L_jk^T;  A_{j,j-1} -= the term k = j-2,
//              L_{j,j-1} = A_{j,j-1} W_{j-1}^T,  S -= L_{j,j-1} L_{j,j-1}^T,
//              L_jj = potrf(S),  W_j = L_jj^-1
//     M(j) holds the whole critical path of column j: once W_{j-1} is there the
//     sub-diagonal tile goes from the TRSM product through shared memory into
//     the diagonal tile's update and its factor, without a trip through global
//     memory and a flag in between.  The terms before run ahead of that; P(j)
//     takes most of them off M(j), which is the longer of the two.
//   * A CTA is four tensor-core warps (DMMA, mma.sync m16n8k4 f64) and a
//     producer warp.  The producer polls for the tiles a task reads and brings
//     16-column chunks of them into a 4-stage ring by cp.async on mbarriers; the
//     others only load fragments and multiply.  Two CTAs per SM: a third costs
//     the registers of the multiplying warps (128 instead of 168) and slows the
//     critical tasks it shares an SM with (n = 16384: 48.6 against 45.2 ms,
//     n = 2048: 0.57 against 0.48).  With the copies and the polls in the
//     multiplying warps two CTAs per SM took 65 ms at n = 16384 and three 53.
//     What bounds it: up to n = 4096 the chain, 13 - 15 us per 64 columns (poll
//     and W 1.5, TRSM and update 4.1, factor 7.2, publish 0.5); above that the
//     DMMA rate (30 TF/s at n = 8192, 32.4 at 16384, of 35.4 for cuBLAS dgemm).
//   * Tasks are handed out by an atomic ticket: M(0), M(1), then per column c
//     T(c+2, c), P(c+2), M(c+2), T(c+3, c), ...: the device form of the
//     reference's priorities (the POTRF/TRSM chain goes out two columns ahead of
//     the rest).  A task waits only on tiles with smaller tickets, which running
//     CTAs hold; so the walk cannot deadlock whatever the residency.
//   * The tiles of a row are finished in column order (tile (i, k) needs every
//     (i, k' < k)), so one counter per row says how many are final.  It is set
//     by a release of one thread after a barrier of the storing warps and read
//     by an acquire of the producer's lane 0, which keeps the value it saw and
//     polls again only past it.  Every wait is bounded by wait_ns of device time;
//     a wait that runs out sets st->timeout, the CTA's copies land and it stops,
//     and the other waiters see the timeout and stop too.
//   * A non-positive pivot is reported LAPACK-style in st->info (1-based
//     global column); the columns before it are final for every row, and the
//     walk still finishes every task (with the inverse's rows from the failure
//     on replaced by identity rows), so nothing waits forever.
#include "common.cuh"
#include "tc_sm100.cuh"

namespace lnb {
namespace dag {

constexpr int TS = 64;              // tile order
constexpr int NT = 128;             // multiplying threads (4 warps)
constexpr int NTHR = NT + 32;       // + the producer warp
constexpr int CPS = 2;              // CTAs per SM
constexpr int BK = 16;              // K chunk
constexpr int ST = 4;               // stages of the chunk ring
constexpr int LDK = TS + 4;         // k-major staged rows (= 4 mod 16 doubles: conflict-free fragments)
constexpr int CHUNK = BK * LDK;     // doubles per staged operand chunk
constexpr int HALF = TS * LDK;      // a whole 64 x 64 tile, k-major
constexpr int PW = 8;               // panel width of the diagonal factor
constexpr uint64_t YIELD_NS = 40000;
constexpr int NBUSY = 256;          // SMs told apart by the busy flags
constexpr int LDX = 10;             // column stride of a panel's 8 x 8 inverse
static_assert(2 * HALF <= 2 * ST * CHUNK, "the epilogue's two tiles fit the ring");
constexpr int XOFF = 2 * ST * CHUNK;   // the panels' inverses, after the ring
constexpr int SMEM = (XOFF + 2 * PW * LDX) * (int)sizeof(double);

struct Args {
    double *A;
    int64_t lda, n;
    int nt, ntasks;
    double *W;              // nt inverses of the diagonal tiles, 64 x 64 column-major each
    int *prog;              // prog[i]: tiles (i, 0 .. prog[i]-1) are final
    int *part;              // part[j]: P(j) is done
    int *busy;              // busy[sm]: a task on that SM is in its critical section
    int *ticket;
    int ticket0;            // first ticket handed out (0; 1 only in the wait self-test)
    lnb_status_t *st;
    long long wait_ns;
};

struct Shared {
    uint64_t full[ST], empty[ST];   // chunk ring
    uint64_t kdone;                 // the sums are read: the ring may be overwritten
    uint64_t sfull, wfull;          // P(j) is done; W is in
    int task, fail;
    int abort;
};
// what a CTA has put through its mbarriers so far (every thread keeps the same)
struct Count {
    int q, kd, sf, wf;
};

// barrier of the four multiplying warps
LNB_DEV void mma_sync() { asm volatile("bar.sync 1, 128;" ::: "memory"); }
LNB_DEV bool mma_sync_and(bool pred)
{
    uint32_t r;
    asm volatile(
        "{\n\t.reg .pred p, q;\n\t"
        "setp.ne.u32 p, %1, 0;\n\t"
        "bar.red.and.pred q, 1, 128, p;\n\t"
        "selp.u32 %0, 1, 0, q;\n\t}"
        : "=r"(r)
        : "r"((uint32_t)pred)
        : "memory");
    return r != 0;
}

// 1/sqrt(d) for a normal d > 0: the approximate instruction, then one step of
// Householder's iteration of third order (A. S. Householder, The Numerical
// Treatment of a Single Nonlinear Equation, 1970) for y^-2 = d:
// y' = y (1 + h/2 + 3 h^2/8), h = 1 - d y^2, whose next term is 5 h^3/16.  With the
// instruction's error below 2^-20 (|h| < 2^-19) that term is 0.02 u; the roundings of
// h and of the last sum are 1.5 u (u = 2^-53).  tests/test_gpu_edges.py holds the
// result to 1.6 u of the exact value and compares it with rsqrt().  Calling rsqrt()
// here instead: n = 200 with one solve 135 us against 125, n = 5003 1.928 ms against
// 1.896.
LNB_DEV double pivot_rsqrt(double d)
{
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(d));
    const double h = fma(-(d * y), y, 1.0);
    return fma(fma(0.375, h, 0.5), y * h, y);
}

// Columns 8p .. 8p+7 of the 64 x 64 tile Sc (column-major, ld LDK) for every
// row from 8p down, and the inverse of their 8 x 8 diagonal block: X =
// inv(L_pp)^T, Xs[c * LDX + r], comes out of the same column steps applied to
// eight identity rows.  A warp holds the eight pivot rows in lanes 0-7 and 48 of
// the other rows (the identity rows first) in the other lanes, two per lane;
// panels 0 and 1 take two warps, which both work on the pivot rows: they meet at
// a barrier between the loads and the first store, because warp 0 stores the
// finished pivot rows where warp 1 loads them.  Every lane tracks the pivots
// (dd): it takes the pivot rows' entries of the column by shuffle before they are
// scaled, so the chain per column is 1/sqrt -> multiply -> fma, and the shuffles
// and the rows' updates run beside it.  The fast form takes every pivot as a finite
// normal positive number and looks at them after the last column (a branch or a select per
// column costs 100 - 270 of its 760 cycles); where one is not, it stores
// nothing and the other form repeats the panel.  Returns the tile column of the
// first non-positive pivot (its column and those after it keep their values),
// 64 if there is none, or -1 (fast form) to ask for the repetition.
LNB_DEV int panel_warps(int p) { return p < 2 ? 2 : 1; }
// every panel warp has loaded its rows (both see the same pivots, so both repeat a panel or
// neither does)
LNB_DEV void panel_loaded(int p)
{
    if (panel_warps(p) == 2) asm volatile("bar.sync 2, 64;" ::: "memory");
}
template <bool FAST>
LNB_DEV int warp_panel8(double *Sc, double *Xs, int p, int w)
{
    const int lane = threadIdx.x & 31;
    const int i0 = lane - PW + 48 * w, i1 = i0 + 24;         // identity rows 0-7, then rows 8p + 8 ..
    const int row0 = PW * p + (lane < PW ? lane : i0), row1 = PW * p + i1;
    const bool ident = lane >= PW && i0 < PW, real0 = !ident && row0 < TS, real1 = lane >= PW && row1 < TS;
    double *col0 = Sc + PW * p * LDK + (real0 ? row0 : 0), *col1 = Sc + PW * p * LDK + (real1 ? row1 : 0);
    double a[PW], b[PW], dd[PW];
#pragma unroll
    for (int k = 0; k < PW; ++k) {
        a[k] = col0[k * LDK];
        b[k] = col1[k * LDK];
        if (!real0) a[k] = ident && k == i0 ? 1.0 : 0.0;
    }
    panel_loaded(p);
#pragma unroll
    for (int k = 0; k < PW; ++k) dd[k] = __shfl_sync(0xffffffffu, a[k], k);
    int fail = TS;
#pragma unroll
    for (int c = 0; c < PW; ++c) {
        double s[PW];
#pragma unroll
        for (int k = c + 1; k < PW; ++k) s[k] = __shfl_sync(0xffffffffu, a[c], k);
        double rs, rt;
        if (FAST) {
            rs = rt = pivot_rsqrt(dd[c]);
        } else {
            if (!(dd[c] > 0.0) && fail == TS) fail = PW * p + c;
            rt = fail == TS ? rsqrt(dd[c]) : 0.0;            // a failed column updates nothing
            rs = fail == TS ? rt : 1.0;
        }
        a[c] *= rs;
        b[c] *= rs;
#pragma unroll
        for (int k = c + 1; k < PW; ++k) {
            s[k] *= rt;
            dd[k] = fma(-s[k], s[k], dd[k]);
            a[k] = fma(-a[c], s[k], a[k]);
            b[k] = fma(-b[c], s[k], b[k]);
        }
    }
    if (FAST) {
        double lo = dd[0];                                   // a NaN fails the comparison below
#pragma unroll
        for (int c = 1; c < PW; ++c) lo = dd[c] < lo || !(dd[c] == dd[c]) ? dd[c] : lo;
        // an infinite pivot makes the ones after it NaN; the last has none after it
        if (!(lo >= 2.2250738585072014e-308 && dd[PW - 1] <= 1.7976931348623157e308)) return -1;   // warp-uniform
    }
    if (ident) {
#pragma unroll
        for (int c = 0; c < PW; ++c) Xs[c * LDX + i0] = a[c];
    } else if (real0 && (w == 0 || lane >= PW)) {
#pragma unroll
        for (int c = 0; c < PW; ++c)
            if (lane >= c) col0[c * LDK] = a[c];
    }
    if (real1) {
#pragma unroll
        for (int c = 0; c < PW; ++c) col1[c * LDK] = b[c];
    }
    return fail;
}
__device__ __noinline__ int warp_panel8_checked(double *Sc, double *Xs, int p, int w)
{
    return warp_panel8<false>(Sc, Xs, p, w);
}

// acc, acc2 += A^T B over the staged rows [k0, k1) (k1 - k0 a multiple of 8): a
// at column m, b at column n of two k-major tiles, eight rows of operands in
// flight and two accumulators against the DMMA latency
LNB_DEV void dot_tile(double (&acc)[4], double (&acc2)[4], const double *Am, const double *Bn, int k0, int k1, int t)
{
    if (k0 >= k1) return;
    const double *ap = Am + (k0 + t) * LDK, *bp = Bn + (k0 + t) * LDK;
    double x0 = ap[0], x1 = ap[8], xb = bp[0], y0 = ap[4 * LDK], y1 = ap[4 * LDK + 8], yb = bp[4 * LDK];
#pragma unroll 1
    for (int k = k0 + 8; k < k1; k += 8) {
        ap += 8 * LDK;
        bp += 8 * LDK;
        const double u0 = ap[0], u1 = ap[8], ub = bp[0], v0 = ap[4 * LDK], v1 = ap[4 * LDK + 8], vb = bp[4 * LDK];
        dmma16x8x4(acc, x0, x1, xb);
        dmma16x8x4(acc2, y0, y1, yb);
        x0 = u0; x1 = u1; xb = ub; y0 = v0; y1 = v1; yb = vb;
    }
    dmma16x8x4(acc, x0, x1, xb);
    dmma16x8x4(acc2, y0, y1, yb);
}

// The CTA: factor the 64 x 64 tile Sc (column-major, ld LDK, lower part) in
// place and store its inverse to Wg (column-major, global).  Bound by latency:
// 64 dependent pivots.  In period p, panel_warps(p) warps factor panel p; the
// others subtract the columns before it from panel p+1 (left-looking, one m16
// row tile per job) and form E - L_p,<p W, rows 8p..8p+7 of the inverse up to the
// factor inv(L_pp), as a transpose so that the tensor cores' N = 8 is the panel
// and M the columns of W (one 16-column tile per job).  Only the last 8 columns'
// two DMMA steps, the product with inv(L_pp) beside them and two barriers sit
// between two panels.  Wr: 64 x LDK
// doubles of scratch (rows of W); the caller zeroes W above its diagonal
// 16 x 16 blocks.  panels: 8, or fewer to run the code on a dummy tile.  Returns the first failed column, or 64.
LNB_DEV int cta_factor64(double *Sc, double *Wr, double *Xs2, double *Wg, int *s_fail, int panels)
{
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5, g = lane >> 2, t = lane & 3;
    auto finish_w = [&](int p, int qt) {             // W rows of panel p, columns of tile qt
        const int q = 16 * qt + g, r = PW * p + 2 * t;
        const double *Xs = Xs2 + (p & 1) * PW * LDX + g * LDX + t, *a = Wr + (PW * p + t) * LDK + q;
        double o[4] = {0.0, 0.0, 0.0, 0.0};
        const double a0 = a[0], a1 = a[8], a2 = a[4 * LDK], a3 = a[4 * LDK + 8], x0 = Xs[0], x1 = Xs[4];
        dmma16x8x4(o, a0, a1, x0);
        dmma16x8x4(o, a2, a3, x1);
        __syncwarp();
        double *wo = Wr + r * LDK + q, *go = Wg + r + TS * q;
        wo[0] = o[0];
        wo[LDK] = o[1];
        wo[8] = o[2];
        wo[LDK + 8] = o[3];
        *reinterpret_cast<double2 *>(go) = make_double2(o[0], o[1]);
        *reinterpret_cast<double2 *>(go + 8 * TS) = make_double2(o[2], o[3]);
    };
    if (tid == 0) *s_fail = TS;
    int p = 0, fail = TS;
#pragma unroll 1
    for (;; ++p) {
        const int np = panel_warps(p);
        const int pn = p + 1, m0 = pn / 2, nupd = (p > 0 && pn < panels) ? 4 - m0 : 0;
        if (w < np) {
            int f = warp_panel8<true>(Sc, Xs2 + (p & 1) * PW * LDX, p, w);
            if (f < 0) f = warp_panel8_checked(Sc, Xs2 + (p & 1) * PW * LDX, p, w);
            if (f < TS && tid == 0) *s_fail = f;
        } else {
            // the longest sums first: W's tile 0, then S, then W's other tiles;
            // a second round goes in reverse order
            const int njobs = nupd + p / 2 + 1, ns = 4 - np;
#pragma unroll 1
            for (int rnd = 0; rnd * ns < njobs; ++rnd) {
                const int job = rnd * ns + ((rnd & 1) ? NT / 32 - 1 - w : w - np);
                if (job >= njobs) continue;
                const bool upd = job > 0 && job <= nupd;
                const int qt = job > 0 ? job - nupd : 0;
                const int m = 16 * (upd ? m0 + job - 1 : qt) + g, pc = PW * (upd ? pn : p), c = pc + 2 * t;
                double *T = (upd ? Sc : Wr) + m;
                double *o0 = T + c * LDK, *o1 = o0 + LDK;
                double acc[4] = {0.0, 0.0, 0.0, 0.0}, acc2[4] = {0.0, 0.0, 0.0, 0.0};
                double e0 = m == c ? 1.0 : 0.0, e1 = m == c + 1 ? 1.0 : 0.0, e2 = m + 8 == c ? 1.0 : 0.0,
                       e3 = m + 8 == c + 1 ? 1.0 : 0.0;
                if (upd) {
                    e0 = o0[0]; e1 = o1[0]; e2 = o0[8]; e3 = o1[8];
                }
                // W is zero above its diagonal
                dot_tile(acc, acc2, T, Sc + pc + g, upd ? 0 : 16 * qt, PW * p, t);
                o0[0] = e0 - (acc[0] + acc2[0]);
                o1[0] = e1 - (acc[1] + acc2[1]);
                o0[8] = e2 - (acc[2] + acc2[2]);
                o1[8] = e3 - (acc[3] + acc2[3]);
            }
        }
        mma_sync();                                  // panel p is final
        fail = *s_fail;
        if (pn == panels || fail < TS) break;
        if (w >= m0) {                               // panel p's own columns
            const int m = 16 * w + g;
            const double *a = Sc + (PW * p + t) * LDK;
            double *o0 = Sc + (PW * pn + 2 * t) * LDK + m, *o1 = o0 + LDK;
            double acc[4] = {0.0, 0.0, 0.0, 0.0}, acc2[4] = {0.0, 0.0, 0.0, 0.0};
            dmma16x8x4(acc, a[m], a[m + 8], a[PW * pn + g]);
            dmma16x8x4(acc2, a[4 * LDK + m], a[4 * LDK + m + 8], a[4 * LDK + PW * pn + g]);
            o0[0] -= acc[0] + acc2[0];
            o1[0] -= acc[1] + acc2[1];
            o0[8] -= acc[2] + acc2[2];
            o1[8] -= acc[3] + acc2[3];
        }
        if (w <= p / 2) finish_w(p, w);
        mma_sync();
    }
    if (w <= p / 2) finish_w(p, w);
    if (fail < TS) {                                 // identity rows from the failure on
        mma_sync();
        for (int idx = tid; idx < TS * TS; idx += NT)
            if ((idx & 63) >= fail) Wg[idx] = (idx & 63) == (idx >> 6) ? 1.0 : 0.0;
    }
    return fail;
}

// ---- the producer warp ---------------------------------------------------------
// rows [r0, r0 + 64) of NC columns from c0 of the column-major matrix as
// dst[kk][m] (k-major), rows at or past n zero-filled, by cp.async of the warp:
// 16 bytes per lane where the matrix is 16-byte aligned, else 8.  (A bulk copy
// per column takes 55 cycles to issue and a proxy fence after each flag; these
// take 7 and none.)
template <int NC>
LNB_DEV void load_cols(double *dst, const double *A, int64_t lda, int64_t n, int64_t r0, int64_t c0, bool vec, int lane)
{
    if (vec) {
        const int64_t r = r0 + 2 * lane;
        const int bytes = r + 1 < n ? 16 : r < n ? 8 : 0;
        const double *g = A + (bytes ? r : 0) + c0 * lda;
        uint32_t d = smem_u32(dst + 2 * lane);
#pragma unroll 8
        for (int c = 0; c < NC; ++c, g += lda, d += LDK * 8)
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(d), "l"(g), "r"(bytes));
    } else {
        const int b0 = r0 + lane < n ? 8 : 0, b1 = r0 + lane + 32 < n ? 8 : 0;
        const double *g0 = A + (b0 ? r0 + lane : 0) + c0 * lda, *g1 = A + (b1 ? r0 + lane + 32 : 0) + c0 * lda;
        uint32_t d = smem_u32(dst + lane);
#pragma unroll 8
        for (int c = 0; c < NC; ++c, g0 += lda, g1 += lda, d += LDK * 8) {
            asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(d), "l"(g0), "r"(b0));
            asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(d + 256), "l"(g1), "r"(b1));
        }
    }
}
// this lane's arrival on bar once its copies so far have landed
LNB_DEV void arrive_copied(uint64_t *bar)
{
    asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}

// spin until min(*f0, *f1) >= target and return it; -1 after wait_ns or once
// another waiter has reported a timeout.  hot: a wait on the critical path,
// without sleeping between the polls.
LNB_DEV int wait_prog(const int *f0, const int *f1, int target, bool hot, const Args &a)
{
    const uint64_t t0 = globaltimer();
    for (int it = 0;; ++it) {
        int v = ld_acquire(f0);
        if (f1 != f0 && v >= target) {
            const int v1 = ld_acquire(f1);
            v = v1 < v ? v1 : v;
        }
        if (v >= target) return v;
        if ((it & 15) == 15) {
            if (ld_acquire(&a.st->timeout) != 0) return -1;
            if ((long long)(globaltimer() - t0) > a.wait_ns) return -1;
        }
        if (!hot) __nanosleep(it < 4 ? 64 : 200);
    }
}

// wait on one of the CTA's mbarriers; false once the CTA has given up or wait_ns
// has passed.  It polls shared memory only: many CTAs wait at once, and polling
// the global status word here slowed every flag of the walk down.
LNB_DEV bool bar_wait(uint64_t *bar, uint32_t parity, long long wait_ns, const Shared &sh)
{
    if (tc::mbar_try_wait(bar, parity)) return true;
    const uint64_t t0 = globaltimer();
    for (int it = 1;; ++it) {
        if (tc::mbar_try_wait(bar, parity)) return true;
        if (*(const volatile int *)&sh.abort) return false;
        if ((it & 63) == 0 && (long long)(globaltimer() - t0) > wait_ns) return false;
    }
}

LNB_DEV void give_up(const Args &a, int site, int item)
{
    if (atomicCAS(&a.st->timeout, 0, site) == 0) a.st->timeout_item = item;
}

// publish: every thread's stores before the caller's barrier, then one
// GPU-scope release by one thread
LNB_DEV void publish(int *flag, int v)
{
    __threadfence();
    asm volatile("st.relaxed.gpu.global.s32 [%0], %1;" ::"l"(flag), "r"(v) : "memory");
}

// L = S W^T for 16 rows per warp: S k-major in Ss (columns p of S), W^T staged
// as Ws[p][q] = W[q][p].  W is lower triangular: column block nb needs p < 8 nb + 8.
LNB_DEV void tile_trsm(double (&o)[8][4], const double *Ss, const double *Ws, int w, int g, int t)
{
#pragma unroll
    for (int nb = 0; nb < 8; ++nb)
#pragma unroll
        for (int q = 0; q < 4; ++q) o[nb][q] = 0.0;
#pragma unroll
    for (int kq = 0; kq < TS / 4; ++kq) {
        const double a0 = Ss[(4 * kq + t) * LDK + 16 * w + g], a1 = Ss[(4 * kq + t) * LDK + 16 * w + g + 8];
#pragma unroll
        for (int nb = 0; nb < 8; ++nb)
            if (nb >= kq / 2) dmma16x8x4(o[nb], a0, a1, Ws[(4 * kq + t) * LDK + 8 * nb + g]);
    }
}

LNB_DEV void prefetch_l2(const double *p)
{
    asm volatile("prefetch.global.L2 [%0];" ::"l"(p));
}
LNB_DEV int *busy_slot(const Args &a)
{
    unsigned smid;
    asm volatile("mov.u32 %0, %%smid;" : "=r"(smid));
    return a.busy + (smid & (NBUSY - 1));
}
LNB_DEV int ld_relaxed(const int *p)
{
    int v;
    asm volatile("ld.relaxed.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

enum Kind { TASK_T, TASK_P, TASK_M };

// the producer's side of one task; false if a wait gave up
LNB_DEV bool produce(const Args &a, Kind kind, int i, int j, bool vec, double *sm, Shared &sh, Count &n)
{
    const int lane = threadIdx.x & 31;
    const bool merged = kind == TASK_M;
    if ((merged && j == 0) || (kind == TASK_P && j < 3)) return true;
    const int jc = kind == TASK_T ? j : j - 1;       // column tile of the product tile
    const int64_t r0 = (int64_t)i * TS, cj = (int64_t)jc * TS;
    const int item = j * a.nt + i;
    const bool hot = kind != TASK_T || i == j + 2;
    const int *pi = a.prog + i, *pj = a.prog + jc;
    int *const busy = busy_slot(a);
    const int nch = (kind == TASK_P ? j - 2 : jc) * (TS / BK);
    const int both = merged ? nch - TS / BK : 0;     // M reads the column tile's rows in the last term only
    int known = 0, held = 0;
    bool ok = true;
    int c = 0;
    for (; c < nch && ok; ++c) {
        // A T task stands back while a task on its SM is in its critical section:
        // the DMMA pipe is shared, and the factor's dependent chain would queue
        // behind this task's products.  Only a hint (nothing waits on it), looked
        // up one chunk ahead and bounded to YIELD_NS.
        if (kind == TASK_T) {
            if (lane == 0) {
                if (held) {
                    const uint64_t t0 = globaltimer();
                    while (ld_relaxed(busy) != 0 && globaltimer() - t0 < YIELD_NS) __nanosleep(100);
                }
                held = ld_relaxed(busy);
            }
            __syncwarp();
        }
        if (merged && c == both && j >= 3) {
            // A_{j,j-1} as P(j) left it
            int v = 0;
            if (lane == 0) v = wait_prog(a.part + j, a.part + j, 1, true, a);
            if (__shfl_sync(0xffffffffu, v, 0) < 0) {
                ok = false;
                break;
            }
            if (lane == 0) tc::mbar_arrive(&sh.sfull);
        }
        if (c / (TS / BK) >= known) {
            if (lane == 0) known = wait_prog(pi, c < both ? pi : pj, c / (TS / BK) + 1, hot, a);
            if (c < both && known > both / (TS / BK)) known = both / (TS / BK);
            known = __shfl_sync(0xffffffffu, known, 0);
            if (known < 0) {
                ok = false;
                break;
            }
        }
        const int s = n.q % ST;
        if (n.q >= ST && !bar_wait(&sh.empty[s], ((n.q / ST) - 1) & 1, a.wait_ns, sh)) ok = false;
        if (!__all_sync(0xffffffffu, ok)) {
            ok = false;
            break;
        }
        double *as = sm + s * 2 * CHUNK;
        const int64_t c0 = (int64_t)c * BK;
        load_cols<BK>(as, a.A, a.lda, a.n, r0, c0, vec, lane);
        if (c >= both) load_cols<BK>(as + CHUNK, a.A, a.lda, a.n, cj, c0, vec, lane);
        arrive_copied(&sh.full[s]);
        ++n.q;
    }
    if (ok && kind != TASK_P) {
        double *V = sm + HALF;
        if (!bar_wait(&sh.kdone, n.kd & 1, 4 * a.wait_ns, sh)) ok = false;
        ok = __all_sync(0xffffffffu, ok);
        ++n.kd;
        if (ok) {
            int v = 0;
            if (lane == 0) {
                if (merged) {
                    // tile (jc, jc-1) is published as M(jc) starts its factor: from
                    // there on this task waits for nothing but that factor
                    v = wait_prog(a.prog + jc, a.prog + jc, jc, true, a);
                    atomicAdd(busy, 1);
                }
                if (v >= 0) v = wait_prog(a.prog + jc, a.prog + jc, jc + 1, hot, a);
            }
            v = __shfl_sync(0xffffffffu, v, 0);
            ok = v >= 0;
            if (ok) {
                load_cols<TS>(V, a.W + (int64_t)jc * TS * TS, TS, TS, 0, 0, true, lane);
                arrive_copied(&sh.wfull);
                ++n.wf;
            }
        }
    }
    if (!ok) {
        if (lane == 0) {
            give_up(a, 31 + (int)kind, item);
            sh.abort = 1;
        }
        cp_async_wait<0>();
    }
    return ok;
}

// the multiplying warps' side of one task; false if a wait gave up
LNB_DEV bool multiply(const Args &a, Kind kind, int i, int j, double *sm, Shared &sh, Count &n)
{
    const bool merged = kind == TASK_M, first = merged && j == 0;
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    const int wm = w >> 1, wn = w & 1, g = lane >> 2, t = lane & 3;
    const int jc = kind == TASK_T ? j : (j > 0 ? j - 1 : 0);
    const int64_t r0 = (int64_t)i * TS, cj = (int64_t)jc * TS;
    const int rows = (int)((a.n - r0) < TS ? (a.n - r0) : TS);
    if (kind == TASK_P && j < 3) return true;
    const int nch = (kind == TASK_P ? j - 2 : jc) * (TS / BK);
    double *S = sm, *V = sm + HALF;

    // the tile's own entries are used after the sum (A - sum keeps the rounding
    // errors at the size of the sum); they come into L2 meanwhile
    {
        const int c = tid >> 1;
        for (int r = 32 * (tid & 1); r < 32 * (tid & 1) + 32 && r < rows; r += 16) {
            if (!first) prefetch_l2(a.A + (r0 + r) + (cj + c) * a.lda);
            if (merged && c < rows) prefetch_l2(a.A + (r0 + r) + (r0 + c) * a.lda);
        }
    }
    bool ok = true;
    auto wait_full = [&](int q) {
        if (ok && !bar_wait(&sh.full[q % ST], (q / ST) & 1, 4 * a.wait_ns, sh)) ok = false;
        return ok;
    };

    double acc[2][4][4];
    auto product = [&](const double *as) {           // acc += A^T B over BK rows of a ring slot
        const double *bs = as + CHUNK + t * LDK + g + wn * 32;
        as += t * LDK + g + wm * 32;
#pragma unroll
        for (int kq = 0; kq < BK / 4; ++kq) {
            const double *ak = as + kq * 4 * LDK, *bk = bs + kq * 4 * LDK;
            const double a0[2] = {ak[0], ak[16]}, a1[2] = {ak[8], ak[24]};
            const double b0[4] = {bk[0], bk[8], bk[16], bk[24]};
#pragma unroll
            for (int mi = 0; mi < 2; ++mi)
#pragma unroll
                for (int ni = 0; ni < 4; ++ni) dmma16x8x4(acc[mi][ni], a0[mi], a1[mi], b0[ni]);
        }
    };
    auto slot = [&](int q) { return sm + (q % ST) * 2 * CHUNK; };
    auto release = [&]() {
        __syncwarp();
        if (lane == 0) tc::mbar_arrive(&sh.empty[n.q % ST]);
        ++n.q;
    };
    // the product tile's entries minus the sum: into S, or back in place.  Sixteen
    // loads in flight: through one pointer the compiler would finish each
    // read-modify-write before the next.
    auto subtract = [&](bool store) {
#pragma unroll
        for (int mi = 0; mi < 2; ++mi) {
            const int r = wm * 32 + mi * 16 + g, c = wn * 32 + 2 * t;
            double *e = a.A + (r0 + r) + (cj + c) * a.lda;
            double v[4][4];
#pragma unroll
            for (int ni = 0; ni < 4; ++ni)
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    const int dr = (q & 2) ? 8 : 0;
                    v[ni][q] = r + dr < rows ? __ldcg(e + dr + (8 * ni + (q & 1)) * a.lda) : 0.0;
                }
#pragma unroll
            for (int ni = 0; ni < 4; ++ni)
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    const int dr = (q & 2) ? 8 : 0;
                    const double x = v[ni][q] - acc[mi][ni][q];
                    if (!store) S[(c + 8 * ni + (q & 1)) * LDK + r + dr] = x;
                    else if (r + dr < rows) e[dr + (8 * ni + (q & 1)) * a.lda] = x;
                }
        }
    };
#pragma unroll
    for (int mi = 0; mi < 2; ++mi)
#pragma unroll
        for (int ni = 0; ni < 4; ++ni)
#pragma unroll
            for (int q = 0; q < 4; ++q) acc[mi][ni][q] = 0.0;

    // M: the diagonal tile's lower 16 x 8 blocks, five per warp (rows 16 bx, then 16 by)
    const int bx = w < 2 ? 3 : 2, by = w == 0 ? 3 : w == 1 ? 0 : w == 2 ? 2 : 1;
    const int nx = w == 1 ? 3 : w == 3 ? 1 : 5, x0 = (w & 1) ? 5 : 0;
    auto drow = [&](int b) { return 16 * (b < nx ? bx : by); };
    auto dcol = [&](int b) { return 8 * (b < nx ? x0 + b : b - nx); };
    double dacc[5][4], da[5][4];                     // its sum, its entries
    auto mma_diag = [&](const double *as) {          // dacc += as^T as over BK rows
#pragma unroll
        for (int kq = 0; kq < BK / 4; ++kq) {
            const double *ak = as + (kq * 4 + t) * LDK + g;
            const double ax0 = ak[16 * bx], ax1 = ak[16 * bx + 8], ay0 = ak[16 * by], ay1 = ak[16 * by + 8];
#pragma unroll
            for (int b = 0; b < 5; ++b) dmma16x8x4(dacc[b], b < nx ? ax0 : ay0, b < nx ? ax1 : ay1, ak[dcol(b)]);
        }
    };
    if (!merged) {
        for (int c = 0; c < nch; ++c) {
            if (!wait_full(n.q)) break;
            product(slot(n.q));
            release();
        }
    } else {
#pragma unroll
        for (int b = 0; b < 5; ++b)
#pragma unroll
            for (int q = 0; q < 4; ++q) dacc[b][q] = 0.0;
        const int early = nch - TS / BK;             // chunks before the term k = j-2
        for (int c = 0; c < early; ++c) {
            if (!wait_full(n.q)) break;
            mma_diag(slot(n.q));
            release();
        }
        if (j >= 3) {                                // the product tile is as P(j) left it
            if (ok && !bar_wait(&sh.sfull, n.sf & 1, 4 * a.wait_ns, sh)) ok = false;
            ++n.sf;
        }
        for (int c = early > 0 ? early : 0; c < nch; ++c) {
            if (!wait_full(n.q)) break;
            product(slot(n.q));
            mma_diag(slot(n.q));
            release();
        }
#pragma unroll
        for (int b = 0; b < 5; ++b)
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const int r = drow(b) + g + ((q & 2) ? 8 : 0), c = dcol(b) + 2 * t + (q & 1);
                da[b][q] = r < rows && r >= c ? __ldcg(a.A + (r0 + r) + (r0 + c) * a.lda) : 0.0;
            }
    }
    if (!first) {
        if (kind != TASK_P) {
            if (lane == 0) tc::mbar_arrive(&sh.kdone);
            ++n.kd;
        }
        if (!mma_sync_and(ok)) return false;         // the ring is free
        subtract(kind == TASK_P);
        if (kind == TASK_P) {
            mma_sync();
            if (tid == 0) publish(a.part + j, 1);
            return true;
        }
    }
    if (!first) {
        // ---- TRSM: L = S W^T ----
        if (ok && !bar_wait(&sh.wfull, n.wf & 1, 4 * a.wait_ns, sh)) ok = false;
        ++n.wf;
        if (!mma_sync_and(ok)) return false;
        double o[8][4];
        tile_trsm(o, S, V, w, g, t);
        if (merged) {
            mma_sync();                              // S is read; L takes its place
#pragma unroll
            for (int nb = 0; nb < 8; ++nb)
#pragma unroll
                for (int q = 0; q < 4; ++q)
                    S[(8 * nb + 2 * t + (q & 1)) * LDK + 16 * w + g + ((q & 2) ? 8 : 0)] = o[nb][q];
            mma_sync();
#pragma unroll 1
            for (int k0 = 0; k0 < TS; k0 += BK) mma_diag(S + k0 * LDK);
        }
#pragma unroll
        for (int nb = 0; nb < 8; ++nb)
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const int r = 16 * w + g + ((q & 2) ? 8 : 0), c = 8 * nb + 2 * t + (q & 1);
                if (r < rows) a.A[(r0 + r) + (cj + c) * a.lda] = o[nb][q];
            }
        if (!merged) {
            mma_sync();
            if (tid == 0) publish(a.prog + i, j + 1);
        }
    }
    if (merged) {
        // ---- the diagonal tile: S, factor, inverse ----
#pragma unroll
        for (int b = 0; b < 5; ++b)
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const int r = drow(b) + g + ((q & 2) ? 8 : 0), c = dcol(b) + 2 * t + (q & 1);
                // padding past the ragged edge factors as the identity
                V[c * LDK + r] = (r < rows && c < rows) ? da[b][q] - dacc[b][q] : (r == c ? 1.0 : 0.0);
            }
        mma_sync();
        if (tid == NT - 1 && j > 0) publish(a.prog + j, j);   // tile (j, j-1), off the factor's warp
        const int f = cta_factor64(V, S, sm + XOFF, a.W + (int64_t)j * TS * TS, &sh.fail, TS / PW);
        mma_sync();
        if (tid == 0) {
            if (f < rows) atomicCAS(&a.st->info, 0, (int)(r0 + f + 1));
            publish(a.prog + j, j + 1);
            if (j > 0) atomicAdd(busy_slot(a), -1);
        }
        // nothing in the walk reads L_jj itself
        for (int idx = tid; idx < TS * TS; idx += NT) {
            const int c = idx / TS, r = idx % TS;
            if (r >= c && r < rows) a.A[(r0 + r) + (r0 + c) * a.lda] = V[c * LDK + r];
        }
    }
    return true;
}

// before an M task: W_j's zeros above the diagonal 16 x 16 blocks; and the
// factor's code, which runs once per M task and rarely twice on one SM (a cold
// run took 2.5 times a warm one), is fetched by three panels of an identity
// tile, ahead of the critical section (W_j gets its own values before it is
// published)
LNB_DEV void warm_factor(const Args &a, int j, double *sm, Shared &sh)
{
    const int tid = threadIdx.x;
    double *Wj = a.W + (int64_t)j * TS * TS;
    for (int q = 16 + (tid >> 3); q < TS; q += NT / 8)
        for (int r = 2 * (tid & 7); r < (q & ~15); r += 16)
            *reinterpret_cast<double2 *>(Wj + TS * q + r) = make_double2(0.0, 0.0);
    if (j == 0) return;
    for (int idx = tid; idx < 3 * PW * LDK; idx += NT) sm[HALF + idx] = idx / LDK == idx % LDK ? 1.0 : 0.0;
    mma_sync();
    cta_factor64(sm + HALF, sm, sm + XOFF, Wj, &sh.fail, 3);
}

__global__ void __launch_bounds__(NTHR, CPS) k_chol_dag_f64(Args a)
{
    extern __shared__ __align__(128) double sm[];
    __shared__ __align__(8) Shared sh;
    const bool vec = ((uintptr_t)a.A % 16 == 0) && (a.lda % 2 == 0);
    const int warp = threadIdx.x >> 5;
    if (threadIdx.x == 0) {
        for (int s = 0; s < ST; ++s) {
            tc::mbar_init(&sh.full[s], 32);
            tc::mbar_init(&sh.empty[s], NT / 32);
        }
        tc::mbar_init(&sh.kdone, NT / 32);
        tc::mbar_init(&sh.sfull, 1);
        tc::mbar_init(&sh.wfull, 32);
        sh.abort = 0;
        tc::fence_mbar_init();
    }
    Count n = {0, 0, 0, 0};
    for (;;) {
        __syncthreads();
        if (*(volatile int *)&sh.abort) break;       // the same for every thread: set before the barrier
        if (threadIdx.x == 0) sh.task = atomicAdd(a.ticket, 1) + a.ticket0;
        __syncthreads();
        const int tk = sh.task;
        if (tk >= a.ntasks) break;
        int i = tk, j = tk;
        Kind kind = TASK_M;
        if (tk >= 2) {
            // column group c holds tickets [2 + c nt - c (c-1)/2, + nt - c)
            int lo = 0, hi = a.nt - 3;
            while (lo < hi) {
                const int mid = (lo + hi + 1) >> 1;
                const int64_t start = 2 + (int64_t)mid * a.nt - (int64_t)mid * (mid - 1) / 2;
                if (start <= tk) lo = mid; else hi = mid - 1;
            }
            const int off = (int)(tk - (2 + (int64_t)lo * a.nt - (int64_t)lo * (lo - 1) / 2));
            kind = off == 1 ? TASK_P : off == 2 ? TASK_M : TASK_T;
            i = lo + 2 + (off > 2 ? off - 2 : 0);
            j = kind == TASK_T ? lo : i;
        }
        if (kind == TASK_M) {
            if (warp < NT / 32) warm_factor(a, j, sm, sh);
            __syncthreads();                         // before the producer's copies
        }
        if (warp == NT / 32 ? !produce(a, kind, i, j, vec, sm, sh, n) : !multiply(a, kind, i, j, sm, sh, n)) {
            if (threadIdx.x == 0) give_up(a, 34, j * a.nt + i);   // stands unless the producer's own wait ran out
            sh.abort = 1;
        }
    }
    cp_async_wait<0>();                              // what the producer issued for a task that gave up
}

}  // namespace dag
}  // namespace lnb

extern "C" int64_t lnb_chol_dag_ints(int64_t n)
{
    const int64_t nt = (n + lnb::dag::TS - 1) / lnb::dag::TS;
    return 2 * nt + 32 + lnb::dag::NBUSY;
}
extern "C" int64_t lnb_chol_dag_w_doubles(int64_t n)
{
    const int64_t nt = (n + lnb::dag::TS - 1) / lnb::dag::TS;
    return nt * lnb::dag::TS * lnb::dag::TS;
}

// sync: lnb_chol_dag_ints(n) ints (zeroed here); W: lnb_chol_dag_w_doubles(n).
// ticket0: first task handed out (0; > 0 only in the wait self-test, where
// skipping the first diagonal tile leaves dependencies that nothing satisfies).
extern "C" int lnb_k_chol_dag_f64(double *A, int64_t lda, int64_t n, double *W, int *sync, lnb_status_t *st,
                                  long long wait_ns, int sms, int ticket0, lnb_stream_t s)
{
    using namespace lnb::dag;
    if (n <= 0) return 0;
    const int64_t nt = (n + TS - 1) / TS;
    if (nt > 8192) return (int)cudaErrorInvalidValue;
    Args a;
    a.A = A; a.lda = lda; a.n = n; a.nt = (int)nt; a.ntasks = (int)(nt < 2 ? nt : 2 + (nt - 2) * (nt + 3) / 2);
    a.W = W; a.ticket = sync; a.ticket0 = ticket0; a.busy = sync + 32; a.prog = sync + 32 + NBUSY; a.part = a.prog + nt; a.st = st; a.wait_ns = wait_ns;
    cudaError_t e = cudaMemsetAsync(sync, 0, (size_t)lnb_chol_dag_ints(n) * sizeof(int), (cudaStream_t)s);
    if (e != cudaSuccess) return (int)e;
    e = cudaFuncSetAttribute(k_chol_dag_f64, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM);
    if (e != cudaSuccess) return (int)e;
    const int grid = (int)(a.ntasks < CPS * sms ? a.ntasks : CPS * sms);
    k_chol_dag_f64<<<grid, NTHR, SMEM, (cudaStream_t)s>>>(a);
    lnb_prof_count(1);
    return (int)cudaGetLastError();
}
