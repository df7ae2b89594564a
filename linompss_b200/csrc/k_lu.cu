// k_lu.cu -- kernels of the tile LU with partial pivoting (lu_main.c, the
// LAPACK dgetrf / dlaswp / dtrsm tasks of lu_kernels.c) and of the general
// solve (gensolv_main.c).
//
//   panel : factor the nb-wide panel A[c0:m, c0:c0+nb] in place with partial
//           pivoting, one CTA of 512 threads (up to 1536 rows of 16 columns) or
//           a cluster of up to 8.  Also composes the panel's row swaps into one
//           permutation of the at most 2 nb rows they touch.
//   apply : the panel's swaps on other columns, and right of the panel the
//           unit-lower solve of its rows and the update of the rows below, on
//           DMMA, in one launch (above 24576 rows the update is a product of its own).
//   laswp : row swaps given as pivots, on any columns.
#include <cooperative_groups.h>
#include <stdlib.h>
#include <limits.h>

#include "common.cuh"
#include "tc_sm100.cuh"

namespace cg = cooperative_groups;

namespace lnb {
namespace lu {

constexpr int MAXNB = 16;
constexpr int MAXCL = 8;
constexpr int PT = 512;                 // threads of a panel CTA
constexpr int PW = PT / 32;

// A panel's swaps as a permutation: row row[e] takes the old contents of row
// src[e], e < cnt; the first nb entries are the panel's own rows.
struct Perm {
    int cnt, pad[3];
    int row[2 * MAXNB], src[2 * MAXNB];
};

// compose the swaps k <-> p[k] (rows counted from the panel's first, p[k] >= k;
// lane k < nk holds p[k]); one warp
LNB_DEV void compose(int p, int nk, Perm *out)
{
    const int lane = threadIdx.x & 31;
    // entry e = lane (panel row e) and e = 32 + lane (a row below)
    int slo = lane, rhi = -1, shi = -1, cnt = nk;
    for (int i = 0; i < nk; ++i) {
        const int pi = __shfl_sync(0xffffffffu, p, i);
        int ip = pi;
        if (pi >= nk) {
            const unsigned hit = __ballot_sync(0xffffffffu, rhi == pi);
            ip = 32 + (hit ? __ffs(hit) - 1 : cnt - nk);
            if (!hit) {
                if (lane == ip - 32) rhi = shi = pi;
                ++cnt;
            }
        }
        const int si = __shfl_sync(0xffffffffu, slo, i);
        const int sp = ip < 32 ? __shfl_sync(0xffffffffu, slo, ip & 31) : __shfl_sync(0xffffffffu, shi, ip & 31);
        if (lane == i) slo = sp;
        if (ip < 32) {
            if (lane == ip) slo = si;
        } else if (lane == ip - 32) {
            shi = si;
        }
    }
    if (lane < nk) { out->row[lane] = lane; out->src[lane] = slo; }
    if (lane < cnt - nk) { out->row[nk + lane] = rhi; out->src[nk + lane] = shi; }
    if (lane == 0) out->cnt = cnt;
}

// Thread t of CTA q holds rows PT RPT q + t + PT i (i < RPT, counted from c0) of
// the columns still to come, a[i][0] the current one: the registers shift down
// by one per column, so the column loop stays rolled.  (Unrolled, its code is
// 40 KB that a panel's SM has never seen, and a cold instruction costs more than
// the column.)  Finished columns of L live in shared memory, where the rows swap
// in place; finished rows of U go straight to A.  Per column: the warps' largest
// entries go to shared memory and an mbarrier, every warp finds the largest of
// them, the warp that holds that row writes it out, and a barrier.  In a cluster
// the CTAs' candidate rows go to each other's shared memory (DSMEM) and that
// barrier is the cluster's.  The next column is updated and searched first: the
// other columns' updates, bound by the FP64 rate, run between the arrival at the
// mbarrier and its completion.
template <int NB, int RPT>
struct PanelSmem {
    double L[NB][PT * RPT];
    double2 prow[2][NB / 2], krow[2][NB / 2];            // the pivot row, the row k
    double2 crow[2][MAXCL][NB], ckrow[2][NB];            // the CTAs' candidates: columns to come, then L
    unsigned long long key[2][PW], ckey[2][MAXCL], bar;
    int idx[2][PW], cidx[2][MAXCL];
    int piv[NB];
};

// the largest key, the smaller index among equals; the same in every lane
LNB_DEV void warp_best(unsigned long long &key, int &idx)
{
    const unsigned hi = (unsigned)(key >> 32), lo = (unsigned)key;
    const unsigned mh = __reduce_max_sync(0xffffffffu, hi);
    const unsigned who = __ballot_sync(0xffffffffu, hi == mh);
    unsigned ml;
    if ((who & (who - 1)) == 0) {                        // one lane has the largest high word
        ml = __shfl_sync(0xffffffffu, lo, __ffs(who) - 1);
        idx = __shfl_sync(0xffffffffu, idx, __ffs(who) - 1);
    } else {
        ml = __reduce_max_sync(0xffffffffu, hi == mh ? lo : 0u);
        idx = __reduce_min_sync(0xffffffffu, hi == mh && lo == ml ? idx : INT_MAX);
    }
    key = (unsigned long long)mh << 32 | ml;
}

// The panel.  Bound by latency: each column is a pivot search over all rows, a row
// broadcast and a rank-1 step, one after another.  A thread holds whole rows of the
// panel in registers (moved down one place per column, so indexes stay constant),
// one block barrier per column (a cluster barrier when the rows need several CTAs),
// and the next column's search runs on its freshly updated values before the rest
// of the row is updated.  16 columns of 1500 rows take 32 us, of 512 rows 17 us
// (32 columns took 130 us by one CTA with the panel in shared memory).
template <int NB, int RPT>
__global__ void __launch_bounds__(PT, 1) k_lu_panel(double *A, int64_t lda, int64_t m, int64_t c0, int nb, int *piv,
                                                    Perm *perm, lnb_status_t *st)
{
    extern __shared__ __align__(16) unsigned char smraw[];
    using SM = PanelSmem<NB, RPT>;
    SM &S = *reinterpret_cast<SM *>(smraw);
    cg::cluster_group cl = cg::this_cluster();
    const int rank = (int)cl.block_rank(), ncl = (int)cl.num_blocks();
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int base = rank * PT * RPT, rows = (int)(m - c0);    // this CTA's first row; rows of the panel
    double a[RPT][NB];
#pragma unroll
    for (int i = 0; i < RPT; ++i) {
        const int r = base + tid + PT * i;
        const double *Ar = A + c0 + (r < rows ? r : 0) + c0 * lda;
#pragma unroll
        for (int j = 0; j < NB; ++j) a[i][j] = (r < rows && j < nb) ? Ar[j * lda] : 0.0;
    }
    unsigned long long key;
    int idx;
    auto search = [&](int k) {                           // the warp's candidate for column k; a NaN counts as zero
        key = 0;
        idx = INT_MAX;
#pragma unroll
        for (int i = 0; i < RPT; ++i) {
            const int r = base + tid + PT * i;
            const double v = fabs(a[i][0]);
            const unsigned long long u = v == v ? (unsigned long long)__double_as_longlong(v) : 0ull;
            if (r >= k && r < rows && (u > key || idx == INT_MAX)) { key = u; idx = r; }
        }
        warp_best(key, idx);
    };
    auto post = [&](int k) {
        if (lane == 0) {
            S.key[k & 1][warp] = key;
            S.idx[k & 1][warp] = idx;
            tc::mbar_arrive((uint64_t *)&S.bar);
        }
    };
    if (tid == 0) {
        tc::mbar_init((uint64_t *)&S.bar, PW);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (ncl > 1) cl.sync(); else __syncthreads();        // also: every CTA of the cluster has started
    search(0);
    post(0);
#pragma unroll 1
    for (int k = 0; k < nb; ++k) {
        const int b = k & 1;
        // 1. the CTA's candidate
        // (the CTA's own 16 warps all arrive; the bound only keeps a spin from
        // lasting, and a panel that met it reports a timeout)
        int spin = 0;
        while (!tc::mbar_try_wait((uint64_t *)&S.bar, b) && spin < (1 << 22)) ++spin;
        int p = lane < PW ? S.idx[b][lane] : INT_MAX;
        key = lane < PW ? S.key[b][lane] : 0ull;
        warp_best(key, p);
        if (spin == 1 << 22) {
            p = rank == 0 ? k : INT_MAX;
            if (lane == 0) atomicCAS(&st->timeout, 0, 41);
        }
        double rp = 1.0 / __longlong_as_double((long long)key);      // 1 / |pivot|, beside the exchange of its row
        // 2. its row and the row k
        const bool own = p != INT_MAX && ((p - base) % PT) >> 5 == warp;
        if (own) {
#pragma unroll
            for (int i = 0; i < RPT; ++i)
                if (base + tid + PT * i == p) {
#pragma unroll
                    for (int j = 0; j < NB; j += 2) S.prow[b][j / 2] = make_double2(a[i][j], a[i][j + 1]);
                }
        }
        if (rank == 0 && warp == 0 && lane == k) {
#pragma unroll
            for (int j = 0; j < NB; j += 2) S.krow[b][j / 2] = make_double2(a[0][j], a[0][j + 1]);
        }
        const double *prow = (const double *)S.prow[b], *krow = (const double *)S.krow[b];
        if (ncl == 1) {
            __syncthreads();
        } else {
            __syncwarp();
            if (own || (p == INT_MAX && warp == 0)) {
                const double v = p == INT_MAX || lane >= NB + k ? 0.0 : lane < NB ? prow[lane] : S.L[lane - NB][p - base];
                for (int q = 0; q < ncl; ++q) {
                    SM *T = cl.map_shared_rank(&S, q);
                    if (lane < 2 * NB) ((double *)T->crow[b][rank])[lane] = v;
                    if (lane == 0) { T->ckey[b][rank] = key; T->cidx[b][rank] = p; }
                }
            }
            if (rank == 0 && warp == 0) {
                const double v = lane >= NB + k ? 0.0 : lane < NB ? krow[lane] : S.L[lane - NB][k];
                for (int q = 0; q < ncl; ++q)
                    if (lane < 2 * NB) ((double *)cl.map_shared_rank(&S, q)->ckrow[b])[lane] = v;
            }
            cl.sync();
            p = lane < ncl ? S.cidx[b][lane] : INT_MAX;
            key = lane < ncl ? S.ckey[b][lane] : 0ull;
            warp_best(key, p);
            rp = 1.0 / __longlong_as_double((long long)key);
            prow = (const double *)S.crow[b][p / (PT * RPT)];
            krow = (const double *)S.ckrow[b];
        }
        const double pv = prow[0];
        // l = a / pv (|a| <= |pv|): one division per column for 1 / pv, then the product
        // with it corrected by its remainder, which rounds as the division does
        // (P. W. Markstein, Computation of Elementary Functions on the IBM RISC
        // System/6000 Processor, IBM J. Res. Dev. 34, 1990); plain divisions where
        // 1 / pv or the remainder may leave the range.  n = 1500: 3.40 ms, with a
        // division per element 3.65.  A zero pivot divides nothing, as in dgetf2.
        const double apv = fabs(pv);
        const bool plain = apv >= 1e-280 && apv <= 1e280;
        rp = copysign(rp, pv);
        // 3. row p takes the old row k
        if (p >= base && p < base + PT * RPT && ((p - base) % PT) >> 5 == warp) {
#pragma unroll
            for (int i = 0; i < RPT; ++i)
                if (base + tid + PT * i == p) {
#pragma unroll
                    for (int j = 0; j < NB; ++j) a[i][j] = krow[j];
                }
        }
        // 4. scale and update the rows below (rows <= k are done: what their
        //    registers and places in L hold is not used)
        double l[RPT];
#pragma unroll
        for (int i = 0; i < RPT; ++i) {
            l[i] = a[i][0];
            if (plain) {
                const double q = l[i] * rp;
                l[i] = fma(fma(-q, pv, l[i]), rp, q);
            } else if (pv != 0.0) {
                l[i] = l[i] / pv;
            }
        }
        {
            const double u = prow[1];
#pragma unroll
            for (int i = 0; i < RPT; ++i) a[i][0] = fma(-l[i], u, a[i][1]);
        }
#pragma unroll
        for (int i = 0; i < RPT; ++i) S.L[k][tid + PT * i] = l[i];
        // the rows of L swap (one warp does it for every column of L); the U row
        if (warp == PW - 1 && lane < k && p != k) {
            if (ncl == 1) {
                const double x = S.L[lane][k];
                S.L[lane][k] = S.L[lane][p];
                S.L[lane][p] = x;
            } else {
                if (rank == 0) S.L[lane][k] = prow[NB + lane];
                if (p >= base && p < base + PT * RPT) S.L[lane][p - base] = krow[NB + lane];
            }
        }
        if (rank == 0 && warp == PW - 2) {
            if (lane < nb - k) A[c0 + k + (c0 + k + lane) * lda] = prow[lane];
            if (lane == 0) {
                S.piv[k] = p;
                piv[c0 + k] = (int)(c0 + p + 1);
                if (pv == 0.0) atomicCAS(&st->info, 0, (int)(c0 + k + 1));
            }
        }
        __syncwarp();
        search(k + 1);
        post(k + 1);
        // the other columns
#pragma unroll
        for (int j = 2; j < NB; ++j) {
            const double u = prow[j];
#pragma unroll
            for (int i = 0; i < RPT; ++i) a[i][j - 1] = fma(-l[i], u, a[i][j]);
        }
#pragma unroll
        for (int i = 0; i < RPT; ++i) a[i][NB - 1] = 0.0;
    }
    __syncthreads();
    if (rank == 0 && warp == 0) compose(lane < nb ? S.piv[lane] : 0, nb, perm);
#pragma unroll
    for (int i = 0; i < RPT; ++i) {
        const int r = base + tid + PT * i;
        double *Ar = A + c0 + (r < rows ? r : 0) + c0 * lda;
#pragma unroll 8
        for (int j = 0; j < NB; ++j)
            if (r > j && r < rows && j < nb) Ar[j * lda] = S.L[j][tid + PT * i];
    }
    if (ncl > 1) cl.sync();                              // no CTA leaves while its smem may be written
}

// The panel's swaps on columns [a0, a1) (left of it) and [b0, b1) (right of it);
// on the right also U = L11^-1 A[c0:c0+nb] and A[below] -= L21 U.  A CTA owns 8
// columns and all their rows, so the swapped rows need no other synchronisation
// than its barriers.  The update is one m16 x n8 DMMA strip of rows per warp at a
// time, U in registers (the B fragments).  Bound by L2: every CTA reads the whole
// panel; with the matrix in L2 and all columns right of the panel updated at once
// a rank-16 step of n = 1500 takes 11 us.
constexpr int AT = 256, AC = 8;
template <int NB>
__global__ void __launch_bounds__(AT) k_lu_apply(double *A, int64_t lda, int64_t m, int64_t c0, int nb,
                                                 const Perm *perm, int64_t a0, int64_t a1, int64_t b0, int64_t b1)
{
    __shared__ double U[NB][AC], L11[NB][NB + 1];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int nleft = (int)((a1 - a0 + AC - 1) / AC);
    const bool left = (int)blockIdx.x < nleft;
    const int64_t j0 = left ? a0 + (int64_t)blockIdx.x * AC : b0 + (int64_t)(blockIdx.x - nleft) * AC;
    const int nc = (int)((left ? a1 : b1) - j0 < AC ? (left ? a1 : b1) - j0 : AC);
    double *X = A + c0 + j0 * lda;                       // this CTA's columns from row c0
    const int cnt = perm->cnt;
    {
        const int e = tid / AC, c = tid % AC;
        const bool act = e < cnt && c < nc;
        double v = 0.0;
        int row = 0;
        if (act) {
            row = perm->row[e];
            v = X[perm->src[e] + c * lda];
        }
        if (!left)
            for (int i = tid; i < nb * nb; i += AT) L11[i % nb][i / nb] = A[c0 + i % nb + (c0 + i / nb) * lda];
        __syncthreads();
        if (act && (left || e >= nb)) X[row + c * lda] = v;
        if (!left && e < NB) U[e][c] = e < nb ? v : 0.0;
    }
    if (left) return;
    static_assert(2 * MAXNB * AC <= AT, "one thread per swapped entry");
    __syncthreads();
    if (warp < AC / 2) {
        // U = L11^-1 U: half a warp per column, lane r holds row r
        const int r = lane & 15, c = 2 * warp + (lane >> 4);
        double x = r < nb ? U[r][c] : 0.0;
        for (int k = 0; k < nb - 1; ++k) {
            const double xk = __shfl_sync(0xffffffffu, x, k, 16);
            if (r > k && r < nb) x = fma(-L11[r][k], xk, x);
        }
        if (r < nb) {
            U[r][c] = x;
            if (c < nc) X[r + c * lda] = x;
        }
    }
    __syncthreads();
    const int g = lane >> 2, t = lane & 3;
    double ub[NB / 4];
#pragma unroll
    for (int q = 0; q < NB / 4; ++q) ub[q] = U[4 * q + t][g];
    const int rows = (int)(m - c0);
    const double *Lp = A + c0 + c0 * lda;
    const bool v0 = 2 * t < nc, v1 = 2 * t + 1 < nc;
    constexpr int SP = 4;                                // strips in flight per warp
    for (int s0 = nb + 16 * warp; s0 < rows; s0 += 16 * SP * (AT / 32)) {
        double la[SP][NB / 4][2], xc[SP][4];
#pragma unroll
        for (int h = 0; h < SP; ++h) {
            const int r = s0 + 16 * h * (AT / 32) + g;
            const bool r0 = r < rows, r1 = r + 8 < rows;
#pragma unroll
            for (int q = 0; q < NB / 4; ++q) {
                const bool kin = 4 * q + t < nb;
                la[h][q][0] = r0 && kin ? Lp[r + (4 * q + t) * lda] : 0.0;
                la[h][q][1] = r1 && kin ? Lp[r + 8 + (4 * q + t) * lda] : 0.0;
            }
            xc[h][0] = r0 && v0 ? X[r + 2 * t * lda] : 0.0;
            xc[h][1] = r0 && v1 ? X[r + (2 * t + 1) * lda] : 0.0;
            xc[h][2] = r1 && v0 ? X[r + 8 + 2 * t * lda] : 0.0;
            xc[h][3] = r1 && v1 ? X[r + 8 + (2 * t + 1) * lda] : 0.0;
        }
#pragma unroll
        for (int h = 0; h < SP; ++h) {
            const int r = s0 + 16 * h * (AT / 32) + g;
#pragma unroll
            for (int q = 0; q < NB / 4; ++q) dmma16x8x4(xc[h], -la[h][q][0], -la[h][q][1], ub[q]);
            if (r < rows && v0) X[r + 2 * t * lda] = xc[h][0];
            if (r < rows && v1) X[r + (2 * t + 1) * lda] = xc[h][1];
            if (r + 8 < rows && v0) X[r + 8 + 2 * t * lda] = xc[h][2];
            if (r + 8 < rows && v1) X[r + 8 + (2 * t + 1) * lda] = xc[h][3];
        }
    }
}

// rows k and piv[k]-1 swap, k = k0..k1-1 in order, on columns [a0, a1) and
// [b0, b1).  Swapping in place would chain every swap's load after the last
// one's store; instead each chunk of up to 32 swaps is first composed into a
// permutation of the (at most 64) rows it touches -- rows[e] receives the old
// contents of row src[e] -- by warp 0 (lane l keeps entries l and l + 32; a
// ballot finds a pivot row among them), then every column thread gathers all
// sources and scatters them: two memory rounds per chunk.
constexpr int SW = 32, SWT = 64;    // 64 threads: the gather buffer is 32 KB of static shared memory
__global__ void __launch_bounds__(SWT) k_laswp(double *A, int64_t lda, int64_t k0, int64_t k1, const int *piv,
                                               int64_t a0, int64_t a1, int64_t b0, int64_t b1)
{
    __shared__ long long rows[2 * SW], src[2 * SW];
    __shared__ int s_cnt;
    __shared__ double vals[2 * SW][SWT];
    const int lane = threadIdx.x & 31;
    const int64_t t = (int64_t)blockIdx.x * SWT + threadIdx.x;
    const int64_t na = a1 > a0 ? a1 - a0 : 0, nbb = b1 > b0 ? b1 - b0 : 0;
    const bool act = t < na + nbb;
    double *col = act ? A + (t < na ? a0 + t : b0 + (t - na)) * lda : A;
    for (int64_t c0 = k0; c0 < k1; c0 += SW) {
        const int nk = (int)(k1 - c0 < SW ? k1 - c0 : SW);
        if (threadIdx.x < 32) {
            const long long pk = lane < nk ? (long long)__ldg(piv + c0 + lane) - 1 : 0;
            // entry e = lane (chunk row c0 + lane) and e = lane + 32 (an extra row)
            long long rlo = c0 + lane, slo = c0 + lane, rhi = -1, shi = -1;
            int cnt = nk;
            for (int i = 0; i < nk; ++i) {
                const long long p = __shfl_sync(0xffffffffu, pk, i);
                int ip;
                if (p < c0 + nk) {
                    ip = (int)(p - c0);
                } else {
                    const unsigned hit = __ballot_sync(0xffffffffu, rhi == p);
                    if (hit) {
                        ip = 32 + __ffs(hit) - 1;
                    } else {
                        ip = 32 + (cnt - nk);
                        if (lane == ip - 32) { rhi = p; shi = p; }
                        ++cnt;
                    }
                }
                // swap src[i] and src[ip]
                const long long si = __shfl_sync(0xffffffffu, slo, i);
                const long long sp = ip < 32 ? __shfl_sync(0xffffffffu, slo, ip & 31)
                                             : __shfl_sync(0xffffffffu, shi, ip & 31);
                if (lane == i) slo = sp;
                if (ip < 32) { if (lane == ip) slo = si; }
                else if (lane == ip - 32) shi = si;
            }
            // pack: entries 0..nk-1, then the extras
            if (lane < nk) { rows[lane] = rlo; src[lane] = slo; }
            if (lane < cnt - nk) { rows[nk + lane] = rhi; src[nk + lane] = shi; }
            if (lane == 0) s_cnt = cnt;
        }
        __syncthreads();
        const int cnt = s_cnt;
        if (act) {
#pragma unroll 8
            for (int i = 0; i < cnt; ++i) vals[i][threadIdx.x] = col[src[i]];
#pragma unroll 8
            for (int i = 0; i < cnt; ++i) col[rows[i]] = vals[i][threadIdx.x];
        }
        __syncthreads();
    }
}

// All of a factorization's swaps as one permutation: row i of the result is old
// row src[i].  The swaps k <-> piv[k]-1 chain, but 32 of them touch at most 64
// rows: every warp composes its chunks against the state before the chunk, and
// the chunks then go through the shared array one after another, a gather and a
// scatter of one warp each (0.15 us a chunk; applying the swaps to the columns in
// turn took 19 us a chunk).
constexpr int CW = 32;              // swaps per chunk
struct Chunk {
    int row[2 * CW], src[2 * CW];   // -1: unused
};
__global__ void __launch_bounds__(1024) k_piv_compose(int n, int k1, const int *piv, int *src)
{
    extern __shared__ __align__(16) int pm[];            // n entries, then one Chunk per warp
    Chunk *ch = reinterpret_cast<Chunk *>(pm + ((n + 3) & ~3));
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nw = blockDim.x >> 5;
    for (int i = tid; i < n; i += blockDim.x) pm[i] = i;
    __syncthreads();
    for (int c0 = 0; c0 < k1; c0 += CW * nw) {
        const int k0 = c0 + CW * warp, nk = k1 - k0 < CW ? k1 - k0 : CW;
        if (nk > 0) {
            const int pk = lane < nk ? piv[k0 + lane] - 1 : 0;
            int slo = k0 + lane, rhi = -1, shi = -1, cnt = 0;
            for (int i = 0; i < nk; ++i) {
                const int p = __shfl_sync(0xffffffffu, pk, i);
                int ip = p - k0;
                if (ip >= nk) {
                    const unsigned hit = __ballot_sync(0xffffffffu, rhi == p);
                    ip = 32 + (hit ? __ffs(hit) - 1 : cnt);
                    if (!hit) {
                        if (lane == cnt) rhi = shi = p;
                        ++cnt;
                    }
                }
                const int si = __shfl_sync(0xffffffffu, slo, i);
                const int sp = ip < 32 ? __shfl_sync(0xffffffffu, slo, ip & 31)
                                       : __shfl_sync(0xffffffffu, shi, ip & 31);
                if (lane == i) slo = sp;
                if (ip < 32) {
                    if (lane == ip) slo = si;
                } else if (lane == ip - 32) {
                    shi = si;
                }
            }
            ch[warp].row[lane] = lane < nk ? k0 + lane : -1;
            ch[warp].src[lane] = slo;
            ch[warp].row[32 + lane] = rhi;
            ch[warp].src[32 + lane] = shi;
        }
        __syncthreads();
        if (warp == 0)
            for (int w = 0; w < nw && c0 + CW * w < k1; ++w) {
                const int r0 = ch[w].row[lane], r1 = ch[w].row[32 + lane];
                const int v0 = r0 >= 0 ? pm[ch[w].src[lane]] : 0, v1 = r1 >= 0 ? pm[ch[w].src[32 + lane]] : 0;
                __syncwarp();
                if (r0 >= 0) pm[r0] = v0;
                if (r1 >= 0) pm[r1] = v1;
                __syncwarp();
            }
        __syncthreads();
    }
    for (int i = tid; i < n; i += blockDim.x) src[i] = pm[i];
}

// T (ld n) = B with its rows permuted; and the copy back
__global__ void __launch_bounds__(256) k_rows_gather(int64_t n, const double *B, int64_t ldb, const int *src, double *T)
{
    const int64_t q = blockIdx.y;
    for (int64_t i = blockIdx.x * 256ll + threadIdx.x; i < n; i += 256ll * gridDim.x) T[i + q * n] = B[src[i] + q * ldb];
}
__global__ void __launch_bounds__(256) k_rows_copy(int64_t n, const double *T, double *B, int64_t ldb)
{
    const int64_t q = blockIdx.y;
    for (int64_t i = blockIdx.x * 256ll + threadIdx.x; i < n; i += 256ll * gridDim.x) B[i + q * ldb] = T[i + q * n];
}

}  // namespace lu
}  // namespace lnb

using namespace lnb::lu;

// Panel width for `rows` rows: NB x RPT = 48 doubles per thread (32 for the
// widest panels of rows), 512 threads per CTA, at most 8 CTAs per cluster: 16
// columns up to 12288 rows, 8 up to 24576, 4 up to 32768; 0 beyond.
extern "C" int lnb_lu_panel_width(int64_t rows)
{
    return rows <= MAXCL * PT * 3 ? 16 : rows <= MAXCL * PT * 6 ? 8 : rows <= MAXCL * PT * 8 ? 4 : 0;
}
extern "C" size_t lnb_lu_perm_bytes(void) { return sizeof(Perm); }

template <int NB, int RPT>
static int launch_panel(double *A, int64_t lda, int64_t m, int64_t c0, int nb, int *piv, Perm *perm, lnb_status_t *st,
                        lnb_stream_t s)
{
    const int64_t rows = m - c0;
    const int ncl = (int)((rows + (int64_t)PT * RPT - 1) / ((int64_t)PT * RPT));
    if (ncl < 1 || ncl > MAXCL || nb > NB) return (int)cudaErrorInvalidValue;
    static_assert(sizeof(PanelSmem<NB, RPT>) <= 227 * 1024, "panel shared memory");
    const cudaError_t e = cudaFuncSetAttribute(k_lu_panel<NB, RPT>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                               (int)sizeof(PanelSmem<NB, RPT>));
    if (e != cudaSuccess) return (int)e;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)ncl);
    cfg.blockDim = dim3(PT);
    cfg.dynamicSmemBytes = sizeof(PanelSmem<NB, RPT>);
    cfg.stream = (cudaStream_t)s;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = (unsigned)ncl;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return (int)cudaLaunchKernelEx(&cfg, k_lu_panel<NB, RPT>, A, lda, m, c0, nb, piv, perm, st);
}

// perm: lnb_lu_perm_bytes() of device memory, for lnb_k_lu_apply_f64
extern "C" int lnb_k_lu_panel_f64(double *A, int64_t lda, int64_t m, int64_t c0, int nb, int *piv, void *perm,
                                  lnb_status_t *st, lnb_stream_t s)
{
    const int64_t rows = m - c0;
    if (rows <= 0 || nb <= 0) return 0;
    const int w = lnb_lu_panel_width(rows);
    if (w == 0 || nb > w) return (int)cudaErrorInvalidValue;
    int e;
    switch (w) {
    case 16:
        /* as few rows per thread as one CTA needs */
        if (rows <= PT) e = launch_panel<16, 1>(A, lda, m, c0, nb, piv, (Perm *)perm, st, s);
        else if (rows <= 2 * PT) e = launch_panel<16, 2>(A, lda, m, c0, nb, piv, (Perm *)perm, st, s);
        else e = launch_panel<16, 3>(A, lda, m, c0, nb, piv, (Perm *)perm, st, s);
        break;
    case 8: e = launch_panel<8, 6>(A, lda, m, c0, nb, piv, (Perm *)perm, st, s); break;
    default: e = launch_panel<4, 8>(A, lda, m, c0, nb, piv, (Perm *)perm, st, s); break;
    }
    lnb_prof_count(1);
    return e;
}

// swaps of the panel at c0 on columns [a0, a1); swaps, solve and update on [b0, b1)
extern "C" int lnb_k_lu_apply_f64(double *A, int64_t lda, int64_t m, int64_t c0, int nb, const void *perm, int64_t a0,
                                  int64_t a1, int64_t b0, int64_t b1, lnb_stream_t s)
{
    const int64_t nl = a1 > a0 ? (a1 - a0 + AC - 1) / AC : 0, nr = b1 > b0 ? (b1 - b0 + AC - 1) / AC : 0;
    if (nl + nr <= 0 || nb <= 0) return 0;
    if (nb > MAXNB) return (int)cudaErrorInvalidValue;
    const unsigned grid = (unsigned)(nl + nr);
    if (a1 < a0) a1 = a0;
    /* Panels of 4 columns (more than 24576 rows): a CTA per 8 columns would run through all the rows for
       a rank-4 step, and inside a 256-column block there are at most 32 such CTAs.  The product's tiles fill
       the chip: 32768 x 256, mean per panel, 119 us in one launch, 7 + 74 as two (panels of 8 columns, 24576 x
       256: 95 in one launch against about 2 x 65). */
    const bool split = lnb_lu_panel_width(m - c0) <= 4 && b1 > b0 && m > c0 + nb;
    const int64_t mu = split ? c0 + nb : m;
    if (nb > 8) k_lu_apply<16><<<grid, AT, 0, (cudaStream_t)s>>>(A, lda, mu, c0, nb, (const Perm *)perm, a0, a1, b0, b1);
    else if (nb > 4) k_lu_apply<8><<<grid, AT, 0, (cudaStream_t)s>>>(A, lda, mu, c0, nb, (const Perm *)perm, a0, a1, b0, b1);
    else k_lu_apply<4><<<grid, AT, 0, (cudaStream_t)s>>>(A, lda, mu, c0, nb, (const Perm *)perm, a0, a1, b0, b1);
    lnb_prof_count(1);
    const int e = (int)cudaGetLastError();
    if (e || !split) return e;
    return lnb_k_gemm_tri_f64('N', 'N', m - c0 - nb, b1 - b0, nb, -1.0, A + (c0 + nb) + c0 * lda, lda, A + c0 + b0 * lda,
                              lda, 1.0, A + (c0 + nb) + b0 * lda, lda, 0, s);
}

extern "C" int lnb_k_laswp_f64(double *A, int64_t lda, int64_t k0, int64_t k1, const int *piv, int64_t a0,
                               int64_t a1, int64_t b0, int64_t b1, lnb_stream_t s)
{
    const int64_t ncols = (a1 > a0 ? a1 - a0 : 0) + (b1 > b0 ? b1 - b0 : 0);
    if (ncols <= 0 || k1 <= k0) return 0;
    k_laswp<<<(unsigned)((ncols + SWT - 1) / SWT), SWT, 0, (cudaStream_t)s>>>(A, lda, k0, k1, piv, a0, a1, b0, b1);
    lnb_prof_count(1);
    return (int)cudaGetLastError();
}

// largest n whose composed permutation fits a block's shared memory (getrs of factors made
// elsewhere may have more rows than the panel kernel takes)
extern "C" int64_t lnb_rows_permute_max(void) { return ((227 * 1024 - 32 * (int64_t)sizeof(Chunk)) / 4) & ~3ll; }

// B (n rows, nrhs columns) takes the swaps k <-> piv[k]-1, k < k1 <= n; src: n
// ints, T: n x tcols doubles of scratch
extern "C" int lnb_k_rows_permute_f64(double *B, int64_t ldb, int64_t n, int64_t nrhs, int64_t k1, const int *piv,
                                      int *src, double *T, int64_t tcols, lnb_stream_t s)
{
    if (n <= 0 || nrhs <= 0 || k1 <= 0) return 0;
    if (n > lnb_rows_permute_max()) return (int)cudaErrorInvalidValue;
    const int smem = (int)((n + 3) & ~3ll) * 4 + 32 * (int)sizeof(Chunk);
    /* the largest of any call, as several host threads may set it */
    cudaError_t e = cudaFuncSetAttribute(k_piv_compose, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
    if (e != cudaSuccess) return (int)e;
    k_piv_compose<<<1, 1024, smem, (cudaStream_t)s>>>((int)n, (int)k1, piv, src);
    lnb_prof_count(1);
    const int64_t step = tcols < 65535 ? tcols : 65535;
    for (int64_t q = 0; q < nrhs; q += step) {
        const int64_t nq = nrhs - q < step ? nrhs - q : step;
        const dim3 grid((unsigned)((n + 255) / 256 < 64 ? (n + 255) / 256 : 64), (unsigned)nq);
        k_rows_gather<<<grid, 256, 0, (cudaStream_t)s>>>(n, B + q * ldb, ldb, src, T);
        k_rows_copy<<<grid, 256, 0, (cudaStream_t)s>>>(n, T, B + q * ldb, ldb);
        lnb_prof_count(2);
    }
    return (int)cudaGetLastError();
}
