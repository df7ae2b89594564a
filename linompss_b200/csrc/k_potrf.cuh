// k_potrf.cuh -- diagonal-tile Cholesky leaf kernel (FP64 and FP32).
//
// Semantics of task_dpotrf / LAPACK potrf 'L' (tasks_potrf.c:20-24) on a
// tile of order bs <= 128, with the info the reference drops reported in
// the status word.  Larger diagonal tiles are factored by the host-side
// nested schedule (leaf POTRF + panel TRSM + update on 128-wide sub-tiles),
// the structure of the reference's nested variant (chol_nrlmain.c).
//
// Bound by latency: one CTA, one tile, a chain of bs pivots.  The whole tile lives
// in shared memory and is factored in 32-column panels:
//   (1) one warp factors the 32 x 32 diagonal block right-looking, a row per lane in
//       registers that move down one place per column (so the loop stays rolled:
//       one-shot code runs at the speed of instruction fetch), and a second warp
//       builds the block's inverse a column behind it, a column per lane; they meet
//       at one 64-thread barrier per column.  Columns are scaled by rsqrt(pivot),
//       the reciprocal LAPACK's potf2 scales by;
//   (2) the rows below the block become b * inv(L_jj)^T: independent dot
//       products, a row per lane and 16 columns per warp, instead of a
//       substitution chain;
//   (3) the rank-32 update of the trailing triangle reads a transposed copy
//       of the panel with vector loads, 4 x 4 outputs per thread.
// FP32, bs = 128: 38 us a tile (68 with all threads on (1), a barrier of the CTA and
// a round through shared memory per column).
// The 32 x 32 inverses are written out (dinv) for the panel TRSM below the
// tile.  After a failed pivot the columns before it are finished for every
// row of the tile, the failing diagonal keeps its updated value, and the
// inverses use the identity past the failure.
#pragma once
#include "common.cuh"

namespace lnb {

constexpr int LEAF = 128;   // max order of a leaf tile
constexpr int LP = 32;      // panel width of the leaf factorization
constexpr int LLI = LP + 4; // row of the block inverse in shared memory

LNB_DEV void leaf_cp_async(float *smem, const float *g)
{
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(smem_u32(smem)), "l"(g));
}
LNB_DEV void leaf_cp_async(double *smem, const double *g) { cp_async8(smem, g, true); }
LNB_DEV float leaf_rsqrt(float x) { return rsqrtf(x); }
LNB_DEV double leaf_rsqrt(double x) { return rsqrt(x); }

// shared memory layout of the leaf (offsets in elements of T, 16-byte aligned)
struct LeafLayout {
    int lds, ldp;
    size_t s_off, p_off, li_off, col_off, total;
};
template <typename T>
__host__ __device__ inline LeafLayout leaf_layout(int bs)
{
    LeafLayout L;
    const int v = 16 / (int)sizeof(T);
    L.lds = bs + 1;
    L.ldp = ((bs + 3) / 4) * 4 + 4;   // 4-row vector reads may run 3 past bs
    L.s_off = 0;
    L.p_off = (((size_t)bs * L.lds + v - 1) / v) * v;
    L.li_off = L.p_off + (size_t)LP * L.ldp;
    L.col_off = L.li_off + (size_t)LP * LLI;
    L.total = L.col_off + 4 * LP + v;
    return L;
}

// the barrier of warps 0 and 1
LNB_DEV void leaf_pair_barrier() { asm volatile("bar.sync 1, 64;" ::: "memory"); }
// 16 consecutive elements, 16-byte aligned
LNB_DEV void leaf_ld16(float (&l)[16], const float *p)
{
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const float4 v = *reinterpret_cast<const float4 *>(p + 4 * i);
        l[4 * i] = v.x; l[4 * i + 1] = v.y; l[4 * i + 2] = v.z; l[4 * i + 3] = v.w;
    }
}
LNB_DEV void leaf_ld16(double (&l)[16], const double *p)
{
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const double2 v = *reinterpret_cast<const double2 *>(p + 2 * i);
        l[2 * i] = v.x; l[2 * i + 1] = v.y;
    }
}
// a[i] <- f(a[i + 1], v[i])
template <typename T, typename F>
LNB_DEV void leaf_shift(T (&a)[LP], const T *v, F f)
{
#pragma unroll
    for (int h = 0; h < LP; h += 16) {
        T l[16];
        leaf_ld16(l, v + h);
#pragma unroll
        for (int i = 0; i < 16; ++i)
            if (h + i + 1 < LP) a[h + i] = f(a[h + i + 1], l[i]);
    }
}

template <typename T>
__global__ void __launch_bounds__(256) k_potrf_leaf(T *A, int64_t lda, int bs, int64_t row0, T *dinv,
                                                    lnb_status_t *st)
{
    extern __shared__ __align__(16) unsigned char sm_raw[];
    const LeafLayout LY = leaf_layout<T>(bs);
    const int LDS = LY.lds, LDP = LY.ldp;
    T *base = reinterpret_cast<T *>(sm_raw);
    T *S = base + LY.s_off;     // S[r * LDS + c] = A[r, c], lower part
    T *Pt = base + LY.p_off;    // Pt[p * LDP + r] = L[r, j0 + p]: the panel below the block, transposed
    T *Li = base + LY.li_off;   // Li[p * LLI + j] = inv(L_jj)[j][p]
    T *Cs = base + LY.col_off;  // [2][LP]: column c below its pivot, over the pivot, by the parity of c
    T *Cu = Cs + 2 * LP;        // [2][LP]: the same as it stands
    T *Rd = Cu + 2 * LP;        // [2]: rsqrt(pivot c), -1 when the pivot is not positive
    __shared__ int fail_col;
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    if (tid == 0) fail_col = bs;

    // the tile arrives by element-wise cp.async, all copies in flight at once
    // (a plain load loop would pay one memory round trip per iteration)
    for (int c = w; c < bs; c += 8)
#pragma unroll
        for (int r = lane; r < LEAF; r += 32)
            if (r >= c && r < bs) leaf_cp_async(S + r * LDS + c, A + (int64_t)r + (int64_t)c * lda);
    cp_async_commit();
    cp_async_wait<0>();
    __syncthreads();

    for (int j0 = 0; j0 < bs; j0 += LP) {
        const int jb = min(LP, bs - j0);
        // ---- (1) factor the jb x jb diagonal block right-looking and build its inverse
        //      X = inv(L_jj) in the same sweep (X = I; for each column c: X[r][:] -=
        //      S[r][c] X[c][:] / d_c for r > c).  Both use the unscaled column over the
        //      pivot, e.g. S[r][cc] -= S[r][c] S[cc][c] / d_c; L's column c and X's row c
        //      are scaled by rsqrt(d_c) (the reciprocal potf2 uses) as they leave.  X lives
        //      in Li (Li[q][r] = X[r][q]). ----
        {
            if (w == 0) {
                T a[LP];                    // a[i] = S[lane][c + i]; above the diagonal not read again
#pragma unroll
                for (int i = 0; i < LP; ++i)
                    a[i] = lane < jb && i <= lane ? S[(j0 + lane) * LDS + j0 + i] : T(0);
                int fc = jb;
                T d = __shfl_sync(0xffffffffu, a[0], 0), inv = leaf_rsqrt(d);
#pragma unroll 1
                for (int c = 0; c < jb; ++c) {
                    const bool ok = d > T(0);                      // potf2 keeps the updated pivot
                    const T a0 = a[0], m = a0 * (inv * inv);
                    T *cs = Cs + (c & 1) * LP, *cu = Cu + (c & 1) * LP;
                    if (lane > c) {
                        cs[lane - c - 1] = m;
                        cu[lane - c - 1] = a0;
                    }
                    if (lane == 0) Rd[c & 1] = ok ? inv : T(-1);
                    // the next pivot: lane c + 1 has all that its diagonal takes, so its
                    // reciprocal root overlaps the exchange of the column
                    const T dn = __shfl_sync(0xffffffffu, a[1] - a0 * m, c + 1);
                    leaf_pair_barrier();
                    if (!ok) { fc = c; break; }
                    const T invn = leaf_rsqrt(dn);
                    leaf_shift(a, cs, [&](T s, T v) { return s - a0 * v; });
                    if (lane >= c && lane < jb) S[(j0 + lane) * LDS + j0 + c] = (lane == c ? d : a0) * inv;
                    d = dn;
                    inv = invn;
                }
                if (fc < jb) {
                    // the columns not reached, as updated so far
#pragma unroll
                    for (int i = 0; i < LP; ++i)
                        if (fc + i <= lane && lane < jb) S[(j0 + lane) * LDS + j0 + fc + i] = a[i];
                    if (lane == 0) {
                        fail_col = j0 + fc;
                        atomicCAS(&st->info, 0, (int)(row0 + j0 + fc + 1));
                    }
                }
            } else if (w == 1) {
                T x[LP];                    // x[i] = X[c + i][lane]
#pragma unroll
                for (int i = 0; i < LP; ++i) x[i] = i == lane ? T(1) : T(0);
                int c = 0;
#pragma unroll 1
                for (; c < jb; ++c) {
                    leaf_pair_barrier();
                    const T inv = Rd[c & 1];
                    if (inv < T(0)) break;
                    const bool in = lane <= c;
                    const T xc = x[0] * (inv * inv);
                    Li[lane * LLI + c] = x[0] * inv;
                    leaf_shift(x, Cu + (c & 1) * LP, [&](T s, T v) { return in ? s - v * xc : s; });
                }
                for (; c < LP; ++c) Li[lane * LLI + c] = c == lane ? T(1) : T(0);   // identity past the end
            }
            __syncthreads();
            if (dinv != nullptr) {
                T *D = dinv + (int64_t)(j0 / LP) * LP * LP;
                for (int idx = tid; idx < LP * LP; idx += blockDim.x) {
                    const int c = idx / LP, r = idx - c * LP;
                    D[r + LP * c] = Li[c * LLI + r];
                }
            }
        }
        // columns of this panel that are final for the rows below
        const int jv = fail_col < bs ? fail_col - j0 : jb;
        // ---- (2) rows below the block: x_r = b_r inv(L_jj)^T; warp: 32 rows, 16 columns.
        //      There are rows only below a full panel (jb = 32), and at most 96 ----
        const int t0 = j0 + jb;
        const int r2 = t0 + 32 * (w >> 1) + lane, c2 = 16 * (w & 1);
        T acc2[16];
        if (t0 + 32 * (w >> 1) < bs) {
            const T *b = S + (r2 < bs ? r2 : bs - 1) * LDS + j0;
#pragma unroll
            for (int s = 0; s < 16; ++s) acc2[s] = T(0);
#pragma unroll 8
            for (int p = 0; p < LP; ++p) {
                const T bp = b[p];
                T l[16];
                leaf_ld16(l, Li + p * LLI + c2);
#pragma unroll
                for (int s = 0; s < 16; ++s) acc2[s] = fma(bp, l[s], acc2[s]);
            }
        }
        __syncthreads();                    // every column's warp has read its rows
        if (r2 < bs) {
#pragma unroll
            for (int s = 0; s < 16; ++s)
                if (c2 + s < jv) {
                    S[r2 * LDS + j0 + c2 + s] = acc2[s];
                    Pt[(c2 + s) * LDP + r2] = acc2[s];
                }
        }
        __syncthreads();
        if (fail_col < bs) break;
        // ---- (3) rank-32 update of the trailing lower triangle, 4x4 per thread ----
        const int tr = bs - t0;
        if (tr > 0) {
            const int nb4 = (tr + 3) / 4, nblk = nb4 * (nb4 + 1) / 2;
            for (int id = tid; id < nblk; id += blockDim.x) {
                int bi = (int)((sqrtf(8.0f * id + 1.0f) - 1.0f) * 0.5f);
                while (bi * (bi + 1) / 2 > id) --bi;
                while ((bi + 1) * (bi + 2) / 2 <= id) ++bi;
                const int bj = id - bi * (bi + 1) / 2;
                const int ra = t0 + 4 * bi, rc = t0 + 4 * bj;
                T acc[4][4];
#pragma unroll
                for (int i = 0; i < 4; ++i)
#pragma unroll
                    for (int j = 0; j < 4; ++j) acc[i][j] = T(0);
#pragma unroll 8
                for (int p = 0; p < LP; ++p) {      // rows below a full panel only
                    T a[4], c[4];
                    if constexpr (sizeof(T) == 4) {
                        const float4 va = *reinterpret_cast<const float4 *>(Pt + p * LDP + ra);
                        const float4 vc = *reinterpret_cast<const float4 *>(Pt + p * LDP + rc);
                        a[0] = va.x; a[1] = va.y; a[2] = va.z; a[3] = va.w;
                        c[0] = vc.x; c[1] = vc.y; c[2] = vc.z; c[3] = vc.w;
                    } else {
                        const double2 va0 = *reinterpret_cast<const double2 *>(Pt + p * LDP + ra);
                        const double2 va1 = *reinterpret_cast<const double2 *>(Pt + p * LDP + ra + 2);
                        const double2 vc0 = *reinterpret_cast<const double2 *>(Pt + p * LDP + rc);
                        const double2 vc1 = *reinterpret_cast<const double2 *>(Pt + p * LDP + rc + 2);
                        a[0] = va0.x; a[1] = va0.y; a[2] = va1.x; a[3] = va1.y;
                        c[0] = vc0.x; c[1] = vc0.y; c[2] = vc1.x; c[3] = vc1.y;
                    }
#pragma unroll
                    for (int i = 0; i < 4; ++i)
#pragma unroll
                        for (int j = 0; j < 4; ++j) acc[i][j] = fma(a[i], c[j], acc[i][j]);
                }
                // the reads first: in one loop each would wait for the write before it
                T *Sb = S + ra * LDS + rc;
#pragma unroll
                for (int i = 0; i < 4; ++i)
#pragma unroll
                    for (int j = 0; j < 4; ++j)
                        if (ra + i < bs && ra + i >= rc + j) acc[i][j] = Sb[i * LDS + j] - acc[i][j];
#pragma unroll
                for (int i = 0; i < 4; ++i)
#pragma unroll
                    for (int j = 0; j < 4; ++j)
                        if (ra + i < bs && ra + i >= rc + j) Sb[i * LDS + j] = acc[i][j];
            }
        }
        __syncthreads();
    }
    __syncthreads();
    // write the lower triangle back (past a failed pivot, the partial state)
#pragma unroll 4
    for (int c = w; c < bs; c += 8) {
        T v[LEAF / 32];
#pragma unroll
        for (int u = 0; u < LEAF / 32; ++u) v[u] = S[min(lane + 32 * u, bs - 1) * LDS + c];
#pragma unroll
        for (int u = 0; u < LEAF / 32; ++u) {
            const int r = lane + 32 * u;
            if (r >= c && r < bs) A[(int64_t)r + (int64_t)c * lda] = v[u];
        }
    }
    // blocks of the tile after a failed panel: identity inverses
    if (dinv != nullptr) {
        const int nq = (bs + LP - 1) / LP;
        const int q0 = fail_col < bs ? fail_col / LP + 1 : nq;
        for (int idx = tid; idx < (nq - q0) * LP * LP; idx += blockDim.x) {
            const int q = q0 + idx / (LP * LP), e = idx % (LP * LP);
            dinv[(int64_t)q * LP * LP + e] = (e % LP == e / LP) ? T(1) : T(0);
        }
    }
}

template <typename T>
inline size_t leaf_smem_bytes(int bs)
{
    return leaf_layout<T>(bs).total * sizeof(T);
}

}  // namespace lnb
