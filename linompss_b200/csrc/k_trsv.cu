// k_trsv.cu -- inverses of diagonal blocks, and blocked triangular solves with an
// FP32 factor and many right-hand sides (k_trsv_chain.cu: few; FP64 factors:
// k_trsm_tiles.cu).
//
// Semantics of bblas_dltrsm (bblas_trsm.h:116-202) and of the two solves of
// dspdsolv_main (spdsolv_main.c:15,17): op(T) X = alpha B with T triangular.
//
// Design: the reference walks block rows with one TRSM task per diagonal
// block and one GEMM task per off-diagonal block.  Here the same task DAG
// runs inside ONE persistent launch:
//   * the h x h diagonal blocks are inverted up front (k_trtri_blocks), so a
//     diagonal "task" is a small GEMM X_j = inv(T_jj) B_j instead of a
//     sequential substitution;
//   * CTAs take work items from an atomic ticket in DAG order (column j's
//     diagonal item, then its off-diagonal updates B_i -= T_ij X_j), so every
//     item only ever waits on items with smaller tickets, which are already
//     held by running CTAs -- the walk cannot deadlock whatever the CTA
//     scheduling order;
//   * an update item stages its T tile in shared memory BEFORE waiting on
//     X_j, so the HBM stream of T overlaps the dependency chain;
//   * every wait is bounded (globaltimer) and reports a timeout instead of
//     hanging.
// Both the tile products use DMMA (m16n8k4 f64).
#include "common.cuh"

namespace lnb {

constexpr int TH = 64;          // block size
constexpr int TLD = TH + 4;     // k-major smem stride (= 4 mod 16 doubles)
constexpr int NRC = 64;         // rhs columns per pass

// ------------------------------------------------------------------------
// inverses of the diagonal blocks
// ------------------------------------------------------------------------
// One CTA inverts one 64 x 64 block, in FP64, stored in the precision of T.  An
// upper block is inverted as the transpose of its transpose.  The four 16 x 16
// diagonal blocks by forward substitution (a thread per column), then twice the
// two-by-two step [A 0; C D]^-1 = [A^-1 0; -D^-1 C A^-1  D^-1], 16 -> 32 -> 64.
// Bound by latency: the substitution over all 64 rows, a thread per column, was
// 64 dependent rows of up to 64 terms and took 56 us (n = 8192, 128 blocks); this takes 20.
constexpr int TI_NT = 256, TI_LD = TH + 1;
// Z (h x h) = sum_k X[.][k] Y[k][.] of h x h blocks (row-major, ld TI_LD), sign s;
// `part` of the CTA's threads: np threads, this one is p
LNB_DEV void ti_product(double *Z, const double *X, const double *Y, int h, double s, int p, int np)
{
    for (int idx = 4 * p; idx < h * h; idx += 4 * np) {
        const int r = idx / h, c = idx % h;
        double z0 = 0.0, z1 = 0.0, z2 = 0.0, z3 = 0.0;
#pragma unroll 8
        for (int k = 0; k < h; ++k) {
            const double x = X[r * TI_LD + k];
            const double *y = Y + k * TI_LD + c;
            z0 = fma(x, y[0], z0);
            z1 = fma(x, y[1], z1);
            z2 = fma(x, y[2], z2);
            z3 = fma(x, y[3], z3);
        }
        double *z = Z + r * TI_LD + c;
        z[0] = s * z0;
        z[1] = s * z1;
        z[2] = s * z2;
        z[3] = s * z3;
    }
}
template <typename TT>
__global__ void __launch_bounds__(TI_NT) k_trtri_blocks(const TT *T, int64_t ldt, int64_t n, char uplo, int unit,
                                                        TT *dinv)
{
    extern __shared__ double smx[];
    double *L = smx, *X = smx + TH * TI_LD;        // row-major: the block (lower), its inverse
    const int q = blockIdx.x, tid = threadIdx.x;
    const int64_t o = (int64_t)q * TH;
    const int qn = (int)((n - o) < TH ? (n - o) : TH);
    const bool lower = uplo == 'L';
    // padding past the ragged edge inverts as the identity
    for (int idx = tid; idx < TH * TH; idx += TI_NT) {
        const int c = idx / TH, r = idx % TH;      // stored row r, column c
        double v = r == c ? 1.0 : 0.0;
        if (r < qn && c < qn && (lower ? r >= c : r <= c) && !(unit && r == c)) v = (double)T[(o + r) + (o + c) * ldt];
        L[lower ? r * TI_LD + c : c * TI_LD + r] = v;
        X[r * TI_LD + c] = 0.0;
    }
    __syncthreads();
    if (tid < TH) {
        const int b0 = tid & ~15, c = tid & 15;    // column c of the 16 x 16 block at b0
        const double *Lb = L + b0 * TI_LD + b0;
        double x[16];
#pragma unroll
        for (int r = 0; r < 16; ++r) {
            double s = r == c ? 1.0 : 0.0, s2 = 0.0;
#pragma unroll
            for (int p = 0; p < r; ++p) {
                if (p & 1) s2 = fma(-Lb[r * TI_LD + p], x[p], s2);
                else s = fma(-Lb[r * TI_LD + p], x[p], s);
            }
            x[r] = (s + s2) / Lb[r * TI_LD + r];
        }
#pragma unroll
        for (int r = 0; r < 16; ++r)
            if (r >= c) X[(b0 + r) * TI_LD + b0 + c] = x[r];
    }
    __syncthreads();
    // (a step whose lower rows are all padding would fill in zeros: skipped)
    if (qn > 16) {
        // 16 -> 32: C A^-1 into the unused upper block of L, then -D^-1 (C A^-1)
        const int b0 = tid < TI_NT / 2 ? 0 : 32, p = tid % (TI_NT / 2);
        double *Lb = L + b0 * TI_LD + b0, *Xb = X + b0 * TI_LD + b0;
        ti_product(Lb + 16, Lb + 16 * TI_LD, Xb, 16, 1.0, p, TI_NT / 2);
        __syncthreads();
        ti_product(Xb + 16 * TI_LD, Xb + 16 * TI_LD + 16, Lb + 16, 16, -1.0, p, TI_NT / 2);
        __syncthreads();
    }
    if (qn > 32) {
        // 32 -> 64
        ti_product(L + 32, L + 32 * TI_LD, X, 32, 1.0, tid, TI_NT);
        __syncthreads();
        ti_product(X + 32 * TI_LD, X + 32 * TI_LD + 32, L + 32, 32, -1.0, tid, TI_NT);
        __syncthreads();
    }
    TT *D = dinv + (int64_t)q * TH * TH;           // column-major
    for (int idx = tid; idx < TH * TH; idx += TI_NT) {
        const int c = idx / TH, r = idx % TH;
        D[idx] = (TT)X[lower ? r * TI_LD + c : c * TI_LD + r];
    }
}

// ------------------------------------------------------------------------
// the DAG walk
// ------------------------------------------------------------------------
template <typename TT>
struct TrsmArgs {
    const TT *T; int64_t ldt; const TT *dinv;
    double *B; int64_t ldb; int64_t n, nrhs;
    int nb; int fwd; int tT;   // tT: op(T) = T^T
    int *ticket, *cnt, *ready;
    lnb_status_t *st; long long wait_ns;
};

// acc(16 rows of warp w, NRC cols) = A(TH x TH, k-major smem) * Bm(TH x NRC, k-major smem)
LNB_DEV void tile_mma(const double *As, const double *Bs, double (&acc)[NRC / 8][4], int w, int g,
                      int t, int ntiles)
{
#pragma unroll
    for (int ni = 0; ni < NRC / 8; ++ni)
#pragma unroll
        for (int q = 0; q < 4; ++q) acc[ni][q] = 0.0;
#pragma unroll 4
    for (int kq = 0; kq < TH / 4; ++kq) {
        const double a0 = As[(kq * 4 + t) * TLD + w * 16 + g];
        const double a1 = As[(kq * 4 + t) * TLD + w * 16 + g + 8];
#pragma unroll
        for (int ni = 0; ni < NRC / 8; ++ni)
            if (ni < ntiles) dmma16x8x4(acc[ni], a0, a1, Bs[(kq * 4 + t) * TLD + ni * 8 + g]);
    }
}

// stage op(T)(block row oi, block col oj) as As[k][m] = op(T)[oi+m][oj+k] (zero-padded)
template <typename TT>
LNB_DEV void stage_tile(const TrsmArgs<TT> &a, double *As, int64_t oi, int in_, int64_t oj, int jn, int tid)
{
    if (!a.tT) {
        for (int idx = tid; idx < TH * TH; idx += 128) {
            const int k = idx / TH, m = idx % TH;
            As[k * TLD + m] = (m < in_ && k < jn) ? (double)a.T[(oi + m) + (oj + k) * a.ldt] : 0.0;
        }
    } else {
        for (int idx = tid; idx < TH * TH; idx += 128) {
            const int m = idx / TH, k = idx % TH;     // op(T)[oi+m][oj+k] = T[oj+k][oi+m]
            As[k * TLD + m] = (m < in_ && k < jn) ? (double)a.T[(oj + k) + (oi + m) * a.ldt] : 0.0;
        }
    }
}

// rhs rows [o, o+rows) x columns [r0, r0+nr) as Bs[k][cc] (k-major), zero-padded
LNB_DEV void stage_rhs(const double *B, int64_t ldb, double *Bs, int64_t o, int rows, int64_t r0, int nr, int tid)
{
    for (int idx = tid; idx < TH * NRC; idx += 128) {
        const int cc = idx / TH, k = idx % TH;
        Bs[k * TLD + cc] = (k < rows && cc < nr) ? __ldcg(&B[(o + k) + (r0 + cc) * ldb]) : 0.0;
    }
}

// Work items in row order of the lower block triangle (virtual rows, reversed
// for an upper op(T)): row ii holds the off-diagonal updates U(ii, jj) for
// jj <= ii-2, then the row item R(ii).  R(ii) absorbs the sub-diagonal update
// U(ii, ii-1) -- the only one on the critical chain --, so the chain per
// block is R(ii-1) -> R(ii): wait X_{ii-1}, one prefetched 64x64 tile product,
// one prefetched inverse product, publish X_ii.  Every item waits only on
// items with smaller tickets.
template <typename TT>
__global__ void __launch_bounds__(128) k_trsm_dag(TrsmArgs<TT> a)
{
    extern __shared__ double smd[];
    double *As = smd;                  // [TH][TLD] tile of op(T)
    double *Ds = smd + TH * TLD;       // [TH][TLD] inverse of the diagonal block
    double *Bs = smd + 2 * TH * TLD;   // [TH][TLD] rhs chunk
    __shared__ int s_item, s_ok;
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5, g = lane >> 2, t = lane & 3;
    const int nb = a.nb;
    const int64_t total = 1 + (int64_t)nb * (nb - 1) / 2;

    while (true) {
        if (tid == 0) s_item = atomicAdd(a.ticket, 1);
        __syncthreads();
        const int64_t item = s_item;
        __syncthreads();
        if (item >= total) break;

        // decode: row ii >= 1 starts at 1 + (ii-1) ii / 2
        int ii = 0, off = 0;
        if (item > 0) {
            ii = (int)((1.0 + sqrt(1.0 + 8.0 * (double)(item - 1))) * 0.5);
            if (ii < 1) ii = 1;
            while (ii > 1 && 1 + (int64_t)(ii - 1) * ii / 2 > item) --ii;
            while (1 + (int64_t)ii * (ii + 1) / 2 <= item) ++ii;
            off = (int)(item - (1 + (int64_t)(ii - 1) * ii / 2));
        }
        const bool row_item = (ii == 0) || (off == ii - 1);
        const int i = a.fwd ? ii : nb - 1 - ii;
        const int64_t oi = (int64_t)i * TH;
        const int in_ = (int)((a.n - oi) < TH ? (a.n - oi) : TH);

        if (row_item) {
            // ---- R(ii): X_i = inv(op T_ii) (B_i - op(T)_{i,p} X_p),  p = previous block ----
            const TT *D = a.dinv + (int64_t)i * TH * TH;
            for (int idx = tid; idx < TH * TH; idx += 128) {
                const int k = idx / TH, m = idx % TH;   // Ds[k][m] = inv(op T_ii)[m][k]
                Ds[k * TLD + m] = a.tT ? D[k + TH * m] : D[m + TH * k];
            }
            const int p = a.fwd ? i - 1 : i + 1;
            const int64_t op_ = (int64_t)p * TH;
            const int pn = ii > 0 ? (int)((a.n - op_) < TH ? (a.n - op_) : TH) : 0;
            if (ii > 0) stage_tile(a, As, oi, in_, op_, pn, tid);
            if (tid == 0) {
                s_ok = wait_geq(&a.cnt[i], ii - 1, a.wait_ns, a.st);
                if (s_ok && ii > 0) s_ok = wait_geq(&a.ready[p], 1, a.wait_ns, a.st);
                if (!s_ok) { atomicCAS(&a.st->timeout, 0, 1); a.st->timeout_item = (int)item; }
            }
            __syncthreads();
            if (!s_ok) return;
            for (int64_t r0 = 0; r0 < a.nrhs; r0 += NRC) {
                const int nr = (int)((a.nrhs - r0) < NRC ? (a.nrhs - r0) : NRC);
                double acc[NRC / 8][4];
                if (ii > 0) {
                    stage_rhs(a.B, a.ldb, Bs, op_, pn, r0, nr, tid);      // X_p
                    __syncthreads();
                    tile_mma(As, Bs, acc, w, g, t, (nr + 7) / 8);
                    __syncthreads();
                } else {
#pragma unroll
                    for (int ni = 0; ni < NRC / 8; ++ni)
#pragma unroll
                        for (int q = 0; q < 4; ++q) acc[ni][q] = 0.0;
                }
                // Bs[m][cc] = B_i - acc   (m becomes k of the inverse product)
#pragma unroll
                for (int ni = 0; ni < NRC / 8; ++ni)
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        const int m = w * 16 + g + ((q & 2) ? 8 : 0);
                        const int cc = ni * 8 + 2 * t + (q & 1);
                        double v = 0.0;
                        if (m < in_ && cc < nr) v = __ldcg(&a.B[(oi + m) + (r0 + cc) * a.ldb]) - acc[ni][q];
                        Bs[m * TLD + cc] = v;
                    }
                __syncthreads();
                tile_mma(Ds, Bs, acc, w, g, t, (nr + 7) / 8);
#pragma unroll
                for (int ni = 0; ni < NRC / 8; ++ni)
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        const int m = w * 16 + g + ((q & 2) ? 8 : 0);
                        const int cc = ni * 8 + 2 * t + (q & 1);
                        if (m < in_ && cc < nr) a.B[(oi + m) + (r0 + cc) * a.ldb] = acc[ni][q];
                    }
                __syncthreads();
            }
            __threadfence();
            __syncthreads();
            if (tid == 0) st_release(&a.ready[i], 1);
        } else {
            // ---- U(ii, jj): B_i -= op(T)_ij X_j ----
            const int jj = off;
            const int j = a.fwd ? jj : nb - 1 - jj;
            const int64_t oj = (int64_t)j * TH;
            const int jn = (int)((a.n - oj) < TH ? (a.n - oj) : TH);
            stage_tile(a, As, oi, in_, oj, jn, tid);
            if (tid == 0) {
                s_ok = wait_geq(&a.ready[j], 1, a.wait_ns, a.st);
                if (!s_ok) { atomicCAS(&a.st->timeout, 0, 2); a.st->timeout_item = (int)item; }
            }
            __syncthreads();
            if (!s_ok) return;
            for (int64_t r0 = 0; r0 < a.nrhs; r0 += NRC) {
                const int nr = (int)((a.nrhs - r0) < NRC ? (a.nrhs - r0) : NRC);
                stage_rhs(a.B, a.ldb, Bs, oj, jn, r0, nr, tid);
                __syncthreads();
                double acc[NRC / 8][4];
                tile_mma(As, Bs, acc, w, g, t, (nr + 7) / 8);
#pragma unroll
                for (int ni = 0; ni < NRC / 8; ++ni)
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        const int m = w * 16 + g + ((q & 2) ? 8 : 0);
                        const int cc = ni * 8 + 2 * t + (q & 1);
                        if (m < in_ && cc < nr) atomicAdd(&a.B[(oi + m) + (r0 + cc) * a.ldb], -acc[ni][q]);
                    }
                __syncthreads();
            }
            __threadfence();
            __syncthreads();
            if (tid == 0) atomicAdd(&a.cnt[i], 1);
        }
    }
}

__global__ void k_scale_f64(double *B, int64_t ldb, int64_t n, int64_t nrhs, double alpha)
{
    const int64_t c = blockIdx.y;
    for (int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; r < n; r += (int64_t)gridDim.x * blockDim.x)
        B[r + c * ldb] *= alpha;
}

}  // namespace lnb

using namespace lnb;

extern "C" int64_t lnb_trsm_sync_ints(int64_t n, int h)
{
    const int64_t nb = (n + h - 1) / h;
    return 4 + 2 * nb;
}

template <typename TT>
static int trtri_blocks(const TT *T, int64_t ldt, int64_t n, int h, char uplo, int unit, TT *dinv, lnb_stream_t s)
{
    if (h != TH) return (int)cudaErrorInvalidValue;
    if (n <= 0) return 0;
    const int64_t nb = (n + TH - 1) / TH;
    const int smem = 2 * TH * (TH + 1) * (int)sizeof(double);
    cudaFuncSetAttribute(k_trtri_blocks<TT>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    k_trtri_blocks<TT><<<(unsigned)nb, TI_NT, smem, s>>>(T, ldt, n, uplo, unit, dinv);
    lnb_prof_count(1);
    return (int)cudaGetLastError();
}

// FP32 T
static int trsm_left(char uplo, char trans, int64_t n, int64_t nrhs, double alpha, const float *T, int64_t ldt,
                     const float *dinv, int h, double *B, int64_t ldb, int *sync, lnb_status_t *st,
                     long long wait_ns, int ticket0, lnb_stream_t s)
{
    if (h != TH) return (int)cudaErrorInvalidValue;
    if (n <= 0 || nrhs <= 0) return 0;
    cudaError_t e;
    if (alpha != 1.0) {
        dim3 grid((unsigned)((n + 255) / 256 < 128 ? (n + 255) / 256 : 128), (unsigned)nrhs);
        k_scale_f64<<<grid, 256, 0, s>>>(B, ldb, n, nrhs, alpha);
        lnb_prof_count(1);
    }
    const int64_t nsync = lnb_trsm_sync_ints(n, h);
    e = cudaMemsetAsync(sync, 0, sizeof(int) * nsync, s);
    if (e != cudaSuccess) return (int)e;
    if (ticket0 != 0) {
        e = cudaMemsetAsync(sync, ticket0 & 0xff, 1, s);  // ticket starts past item 0
        if (e != cudaSuccess) return (int)e;
    }
    if (nrhs <= 8)
        return lnb_k_trsm_chain_f32(uplo, trans, n, nrhs, T, ldt, dinv, B, ldb, sync, st, wait_ns, s);
    TrsmArgs<float> a;
    a.T = T; a.ldt = ldt; a.dinv = dinv; a.B = B; a.ldb = ldb; a.n = n; a.nrhs = nrhs;
    a.nb = (int)((n + TH - 1) / TH);
    const bool lowerop = (uplo == 'L') == (trans == 'N');
    a.fwd = lowerop ? 1 : 0;
    a.tT = (trans == 'T') ? 1 : 0;
    a.ticket = sync; a.cnt = sync + 4; a.ready = sync + 4 + a.nb;
    a.st = st; a.wait_ns = wait_ns;
    int dev = 0, sms = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const int64_t items = 1 + (int64_t)a.nb * (a.nb - 1) / 2;
    int64_t grid = (int64_t)sms * 4;
    if (grid > items) grid = items;
    const int smem = 3 * TH * TLD * (int)sizeof(double);
    cudaFuncSetAttribute(k_trsm_dag<float>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    k_trsm_dag<float><<<(unsigned)grid, 128, smem, s>>>(a);
    lnb_prof_count(1);
    return (int)cudaGetLastError();
}

extern "C" int lnb_k_trtri_blocks_f64(const double *T, int64_t ldt, int64_t n, int h, char uplo, int unit,
                                      double *dinv, lnb_stream_t s)
{
    return trtri_blocks<double>(T, ldt, n, h, uplo, unit, dinv, s);
}
extern "C" int lnb_k_trtri_blocks_f32(const float *T, int64_t ldt, int64_t n, int h, char uplo, int unit,
                                      float *dinv, lnb_stream_t s)
{
    return trtri_blocks<float>(T, ldt, n, h, uplo, unit, dinv, s);
}
extern "C" int lnb_k_trsm_left_f32(char uplo, char trans, int64_t n, int64_t nrhs, double alpha, const float *T,
                                   int64_t ldt, const float *dinv, int h, double *B, int64_t ldb, int *sync,
                                   lnb_status_t *st, long long wait_ns, int ticket0, lnb_stream_t s)
{
    return trsm_left(uplo, trans, n, nrhs, alpha, T, ldt, dinv, h, B, ldb, sync, st, wait_ns, ticket0, s);
}
