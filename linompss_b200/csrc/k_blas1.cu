// k_blas1.cu -- FP64 vector kernels of the refinement loop (HBM-bound).
//
// Semantics: bblas_dgemm used as a matvec (itref.c:1019,1094 and
// bblas_dgemm_prior itref.c:803), bblas_ddot (task_dot.c:30-59),
// bblas_dcpaxpy_comb (task_axpy.c:154-176), bblas_extm_daxpy
// (task_axpy.c:89-97), bblas_sdcpaxpy (task_axpy.c:111-119).
//
// All reductions are deterministic: fixed-shape per-CTA partial sums
// followed by a single-CTA reduction in a fixed order, so repeated runs give
// bit-identical iterates (the refinement decisions do not depend on atomics'
// arrival order).
#include "common.cuh"

namespace lnb {

constexpr int GV_ROWS = 256;    // rows per CTA (one per thread)
constexpr int GV_COLS = 64;     // columns per CTA slab (256 left 36 CTAs at n = 1500: 37 us)

// partial[s][r] = sum_{c in slab s} A[r, c] x[c]
__global__ void __launch_bounds__(GV_ROWS) k_gemv_partial(const double *__restrict__ A, int64_t lda,
                                                          int64_t m, int64_t n,
                                                          const double *__restrict__ x,
                                                          double *__restrict__ part)
{
    __shared__ double xs[GV_COLS];
    const int64_t r = (int64_t)blockIdx.x * GV_ROWS + threadIdx.x;
    const int64_t c0 = (int64_t)blockIdx.y * GV_COLS;
    const int nc = (int)((n - c0) < GV_COLS ? (n - c0) : GV_COLS);
    if (threadIdx.x < nc) xs[threadIdx.x] = x[c0 + threadIdx.x];
    __syncthreads();
    if (r >= m) return;
    const double *a = A + r + c0 * lda;
    double s0 = 0.0, s1 = 0.0, s2 = 0.0, s3 = 0.0;
    int c = 0;
    for (; c + 4 <= nc; c += 4) {
        s0 = fma(__ldcs(a + (int64_t)(c + 0) * lda), xs[c + 0], s0);
        s1 = fma(__ldcs(a + (int64_t)(c + 1) * lda), xs[c + 1], s1);
        s2 = fma(__ldcs(a + (int64_t)(c + 2) * lda), xs[c + 2], s2);
        s3 = fma(__ldcs(a + (int64_t)(c + 3) * lda), xs[c + 3], s3);
    }
    for (; c < nc; ++c) s0 = fma(__ldcs(a + (int64_t)c * lda), xs[c], s0);
    part[(int64_t)blockIdx.y * m + r] = (s0 + s1) + (s2 + s3);
}

// y[r] = beta*y[r] + alpha*sum_s part[s][r]; optionally dpart[blk] = sum y[r]*w[r]
__global__ void __launch_bounds__(256) k_gemv_finish(const double *__restrict__ part, int nslab, int64_t m,
                                                     double alpha, double beta, const double *yin,
                                                     double *y, const double *w, double *dpart)
{
    __shared__ double red[256];
    const int64_t r = (int64_t)blockIdx.x * 256 + threadIdx.x;
    double prod = 0.0;
    if (r < m) {
        double s = 0.0;
        for (int q = 0; q < nslab; ++q) s += part[(int64_t)q * m + r];
        double v = alpha * s;
        if (beta != 0.0) v += beta * yin[r];
        y[r] = v;
        if (w) prod = v * w[r];
    }
    if (!dpart) return;
    red[threadIdx.x] = prod;
    __syncthreads();
    for (int o = 128; o > 0; o >>= 1) {
        if (threadIdx.x < o) red[threadIdx.x] += red[threadIdx.x + o];
        __syncthreads();
    }
    if (threadIdx.x == 0) dpart[blockIdx.x] = red[0];
}

// dpart[blk] = sum over the block's 256*ITEMS elements of x*y
__global__ void __launch_bounds__(256) k_dot_partial(const double *x, const double *y, int64_t n,
                                                     double *dpart)
{
    __shared__ double red[256];
    const int64_t base = (int64_t)blockIdx.x * 2048;
    double s = 0.0;
    for (int i = threadIdx.x; i < 2048; i += 256) {
        const int64_t r = base + i;
        if (r < n) s = fma(x[r], y[r], s);
    }
    red[threadIdx.x] = s;
    __syncthreads();
    for (int o = 128; o > 0; o >>= 1) {
        if (threadIdx.x < o) red[threadIdx.x] += red[threadIdx.x + o];
        __syncthreads();
    }
    if (threadIdx.x == 0) dpart[blockIdx.x] = red[0];
}

// out[0] = sum of nparts partials (one CTA, fixed order)
__global__ void __launch_bounds__(256) k_sum(const double *dpart, int nparts, double *out)
{
    __shared__ double red[256];
    double s = 0.0;
    for (int i = threadIdx.x; i < nparts; i += 256) s += dpart[i];
    red[threadIdx.x] = s;
    __syncthreads();
    for (int o = 128; o > 0; o >>= 1) {
        if (threadIdx.x < o) red[threadIdx.x] += red[threadIdx.x + o];
        __syncthreads();
    }
    if (threadIdx.x == 0) out[0] = red[0];
}

// CG step update with the reference's coefficients (itref.c:806, task_axpy.c:154-176):
//   f = num[0]/den[0];  x += f p;  r += (-1*f) tmp;  partial <r,r>
__global__ void __launch_bounds__(256) k_cg_xr(int64_t n, const double *num, const double *den,
                                               const double *p, const double *tmp, double *x, double *r,
                                               double *dpart)
{
    __shared__ double red[256];
    const double f = num[0] / den[0];
    const int64_t base = (int64_t)blockIdx.x * 2048;
    double s = 0.0;
    for (int i = threadIdx.x; i < 2048; i += 256) {
        const int64_t q = base + i;
        if (q < n) {
            x[q] = x[q] + f * p[q];
            const double rv = r[q] + (-1.0 * f) * tmp[q];
            r[q] = rv;
            s = fma(rv, rv, s);
        }
    }
    red[threadIdx.x] = s;
    __syncthreads();
    for (int o = 128; o > 0; o >>= 1) {
        if (threadIdx.x < o) red[threadIdx.x] += red[threadIdx.x + o];
        __syncthreads();
    }
    if (threadIdx.x == 0) dpart[blockIdx.x] = red[0];
}

// direction update.  mode 0: the reference's executed recurrence p = r; p += 1*p
// (task_axpy.c:89-97 with X == Z, factor alpha1[i]/alpha1[iprev] == 1);
// mode 1: textbook CG, p = z + (num/den) p.
__global__ void k_cg_p(int64_t n, int mode, const double *num, const double *den, const double *r,
                       double *p)
{
    const double beta = mode ? num[0] / den[0] : 0.0;
    for (int64_t q = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; q < n; q += (int64_t)gridDim.x * blockDim.x) {
        if (mode) {
            p[q] = r[q] + beta * p[q];
        } else {
            double v = r[q];
            v = v + 1.0 * v;
            p[q] = v;
        }
    }
}

// ---- dcg_pure as one launch ---------------------------------------------------
// The whole solve of itref.c:690-925 (dense, s = 1) in one cooperative launch, one
// CTA per SM, one grid barrier per step.  Every CTA keeps r and the direction p in
// shared memory and does the vector work of a step redundantly, in the same order,
// so the scalars agree to the last bit without being exchanged; only the product
// A p is shared out, in tiles of 32 rows x a slab of columns, each leaving 32
// partial sums.  All sums have a fixed shape: repeated runs are bit-identical.
// Bound by latency up to a few thousand unknowns (n = 1500: 9 us a step, the matrix
// in L2; as four launches and a host read per step it took 60), by the read of A
// above.
constexpr int CG_NT = 512, CG_NW = CG_NT / 32, CG_RG = 32;

struct CgArgs {
    int64_t n;
    const double *A; int64_t lda;
    const double *b;
    double *x;                  // start vector in, iterate out
    double *part;               // 2 x cs x n partial sums, by step parity
    int cs, steps;
    double tol;
    int *bar;                   // grid barrier counter (zeroed)
    int *out;                   // [0] steps done, [1] converged
    lnb_status_t *st;
    long long wait_ns;
};

// sum over the CTA, the same in every thread
LNB_DEV double cg_sum(double v, double *red)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    __syncthreads();
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
    __syncthreads();
    double s = 0.0;
#pragma unroll
    for (int w = 0; w < CG_NW; ++w) s += red[w];
    return s;
}

// every CTA's stores before it are visible after it; false: the wait ran out
LNB_DEV bool cg_barrier(const CgArgs &a, int phase, int *s_ok)
{
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        atomicAdd(a.bar, 1);
        const int target = (phase + 1) * (int)gridDim.x;
        const uint64_t t0 = globaltimer();
        int ok = 1;
        for (int it = 1; ld_acquire(a.bar) < target; ++it)
            if ((it & 63) == 0 && ((long long)(globaltimer() - t0) > a.wait_ns || ld_acquire(&a.st->timeout) != 0)) {
                atomicCAS(&a.st->timeout, 0, 61);
                ok = 0;
                break;
            }
        *s_ok = ok;
    }
    __syncthreads();
    return *s_ok != 0;
}

// part = A v (v in shared memory), this CTA's tiles
LNB_DEV void cg_product(const CgArgs &a, const double *v, double *part, double *tile)
{
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int rgs = (int)((a.n + CG_RG - 1) / CG_RG);
    const int64_t wc = (a.n + a.cs - 1) / a.cs;
    for (int t = blockIdx.x; t < rgs * a.cs; t += gridDim.x) {
        const int rg = t % rgs, sl = t / rgs;
        const int64_t r = (int64_t)rg * CG_RG + lane, c1 = (sl + 1) * wc < a.n ? (sl + 1) * wc : a.n;
        const double *Ar = a.A + (r < a.n ? r : 0);
        double s0 = 0.0, s1 = 0.0, s2 = 0.0, s3 = 0.0;
        int64_t c = sl * wc + w;
        for (; c + 7 * CG_NW < c1; c += 8 * CG_NW) {
            double e[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) e[u] = __ldg(Ar + (c + u * CG_NW) * a.lda);
            s0 = fma(e[0], v[c], s0);
            s1 = fma(e[1], v[c + CG_NW], s1);
            s2 = fma(e[2], v[c + 2 * CG_NW], s2);
            s3 = fma(e[3], v[c + 3 * CG_NW], s3);
            s0 = fma(e[4], v[c + 4 * CG_NW], s0);
            s1 = fma(e[5], v[c + 5 * CG_NW], s1);
            s2 = fma(e[6], v[c + 6 * CG_NW], s2);
            s3 = fma(e[7], v[c + 7 * CG_NW], s3);
        }
        for (; c < c1; c += CG_NW) s0 = fma(__ldg(Ar + c * a.lda), v[c], s0);
        tile[w * CG_RG + lane] = (s0 + s1) + (s2 + s3);
        __syncthreads();
        if (w == 0 && r < a.n) {
            double s = 0.0;
#pragma unroll
            for (int q = 0; q < CG_NW; ++q) s += tile[q * CG_RG + lane];
            part[sl * a.n + r] = s;
        }
        __syncthreads();
    }
}

__global__ void __launch_bounds__(CG_NT, 1) k_dcg(CgArgs a)
{
    extern __shared__ __align__(16) double smc[];
    double *p = smc, *r = smc + a.n;
    __shared__ double red[CG_NW], tile[CG_NW * CG_RG];
    __shared__ int s_ok;
    const int tid = threadIdx.x, n = (int)a.n;
    // a step writes one half of part while the step before may still be read
    int phase = 0;
    auto part = [&]() { return a.part + (phase & 1) * (int64_t)a.cs * n; };
    auto product_at = [&](const double *pt, int i) {
        double s = 0.0;
        for (int q = 0; q < a.cs; ++q) s += __ldcg(pt + (int64_t)q * n + i);
        return s;
    };
    // r = b - A x;  p = r;  alpha1 = <r, r>
    double bb = 0.0;
    for (int i = tid; i < n; i += CG_NT) {
        p[i] = a.x[i];
        bb = fma(a.b[i], a.b[i], bb);
    }
    bb = cg_sum(bb, red);
    const double norm_b = sqrt(bb);
    const double *pt = part();
    cg_product(a, p, part(), tile);
    if (!cg_barrier(a, phase++, &s_ok)) return;
    double alpha1 = 0.0;
    for (int i = tid; i < n; i += CG_NT) {
        const double v = a.b[i] - product_at(pt, i);
        r[i] = p[i] = v;
        alpha1 = fma(v, v, alpha1);
    }
    alpha1 = cg_sum(alpha1, red);
    // the CTAs share out x; nobody reads it before the end
    const int xs = (n + gridDim.x - 1) / gridDim.x, x0 = blockIdx.x * xs, x1 = x0 + xs < n ? x0 + xs : n;
    int k = 0, done = 0;
    for (; k < a.steps && !done; ++k) {
        pt = part();
        cg_product(a, p, part(), tile);
        if (!cg_barrier(a, phase++, &s_ok)) return;
        // alpha2 = <A p, p>
        double alpha2 = 0.0;
        for (int i = tid; i < n; i += CG_NT) alpha2 = fma(product_at(pt, i), p[i], alpha2);
        alpha2 = cg_sum(alpha2, red);
        const double f = alpha1 / alpha2;
        // x += f p, r -= f A p, alpha1 = <r, r>, and the direction as the reference forms it
        for (int i = x0 + tid; i < x1; i += CG_NT) a.x[i] = a.x[i] + f * p[i];
        __syncthreads();
        alpha1 = 0.0;
        for (int i = tid; i < n; i += CG_NT) {
            const double v = r[i] + (-1.0 * f) * product_at(pt, i);
            r[i] = v;
            p[i] = v + 1.0 * v;
            alpha1 = fma(v, v, alpha1);
        }
        alpha1 = cg_sum(alpha1, red);
        done = sqrt(alpha1) / norm_b <= a.tol;
    }
    if (blockIdx.x == 0 && tid == 0) {
        a.out[0] = k;
        a.out[1] = done;
    }
}

// z = y + a*x   (bblas_sdcpaxpy / task_sdcpaxpy)
__global__ void k_axpy3(int64_t n, double a, const double *x, const double *y, double *z)
{
    for (int64_t q = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; q < n; q += (int64_t)gridDim.x * blockDim.x)
        z[q] = y[q] + a * x[q];
}

}  // namespace lnb

using namespace lnb;

extern "C" int64_t lnb_gemv_part_doubles(int64_t m, int64_t n)
{
    return ((n + GV_COLS - 1) / GV_COLS) * m;
}
extern "C" int64_t lnb_dot_part_doubles(int64_t n) { return (n + 2047) / 2048 + 1; }

// y = alpha A x + beta yin  (A m x n); if w: dot_out = <y, w> (device scalar)
extern "C" int lnb_k_gemv_f64(int64_t m, int64_t n, double alpha, const double *A, int64_t lda,
                              const double *x, double beta, const double *yin, double *y,
                              const double *w, double *dot_out, double *part, double *dpart,
                              lnb_stream_t s)
{
    if (m <= 0) return 0;
    const int nslab = (int)((n + GV_COLS - 1) / GV_COLS);
    if (n > 0) {
        dim3 grid((unsigned)((m + GV_ROWS - 1) / GV_ROWS), (unsigned)nslab);
        k_gemv_partial<<<grid, GV_ROWS, 0, s>>>(A, lda, m, n, x, part);
        lnb_prof_count(1);
    }
    const int nblk = (int)((m + 255) / 256);
    k_gemv_finish<<<nblk, 256, 0, s>>>(part, n > 0 ? nslab : 0, m, alpha, beta, yin, y, w,
                                       dot_out ? dpart : nullptr);
    lnb_prof_count(1);
    if (dot_out) {
        k_sum<<<1, 256, 0, s>>>(dpart, nblk, dot_out);
        lnb_prof_count(1);
    }
    return (int)cudaGetLastError();
}

extern "C" int lnb_k_dot_f64(int64_t n, const double *x, const double *y, double *out, double *dpart,
                             lnb_stream_t s)
{
    const int nblk = (int)((n + 2047) / 2048);
    if (nblk > 0) {
        k_dot_partial<<<nblk, 256, 0, s>>>(x, y, n, dpart);
        lnb_prof_count(1);
    }
    k_sum<<<1, 256, 0, s>>>(dpart, nblk, out);
    lnb_prof_count(1);
    return (int)cudaGetLastError();
}

extern "C" int lnb_k_cg_xr_f64(int64_t n, const double *num, const double *den, const double *p,
                               const double *tmp, double *x, double *r, double *rr_out, double *dpart,
                               lnb_stream_t s)
{
    const int nblk = (int)((n + 2047) / 2048);
    if (nblk > 0) {
        k_cg_xr<<<nblk, 256, 0, s>>>(n, num, den, p, tmp, x, r, dpart);
        lnb_prof_count(1);
    }
    k_sum<<<1, 256, 0, s>>>(dpart, nblk, rr_out);
    lnb_prof_count(1);
    return (int)cudaGetLastError();
}

extern "C" int lnb_k_cg_p_f64(int64_t n, int mode, const double *num, const double *den, const double *r,
                              double *p, lnb_stream_t s)
{
    if (n <= 0) return 0;
    k_cg_p<<<(unsigned)((n + 255) / 256 < 1184 ? (n + 255) / 256 : 1184), 256, 0, s>>>(n, mode, num, den, r, p);
    lnb_prof_count(1);
    return (int)cudaGetLastError();
}

extern "C" int lnb_k_axpy3_f64(int64_t n, double a, const double *x, const double *y, double *z,
                               lnb_stream_t s)
{
    if (n <= 0) return 0;
    k_axpy3<<<(unsigned)((n + 255) / 256 < 1184 ? (n + 255) / 256 : 1184), 256, 0, s>>>(n, a, x, y, z);
    lnb_prof_count(1);
    return (int)cudaGetLastError();
}

// one cooperative launch of dcg_pure: the largest n it takes (r and p in shared memory)
extern "C" int64_t lnb_dcg_max_n(void) { return 12288; }
extern "C" int64_t lnb_dcg_part_doubles(int64_t n, int sms)
{
    const int64_t rgs = (n + CG_RG - 1) / CG_RG;
    return 2 * n * (rgs < sms ? sms / rgs : 1);
}
// part: lnb_dcg_part_doubles(n, sms); sync: 64 ints (zeroed here; [32] steps done and
// [33] converged on return)
extern "C" int lnb_k_dcg_f64(int64_t n, const double *A, int64_t lda, const double *b, double *x, double tol, int steps,
                             double *part, int *sync, lnb_status_t *st, long long wait_ns, int sms, lnb_stream_t s)
{
    if (n <= 0 || n > lnb_dcg_max_n()) return (int)cudaErrorInvalidValue;
    CgArgs a;
    a.n = n; a.A = A; a.lda = lda; a.b = b; a.x = x; a.part = part; a.steps = steps; a.tol = tol;
    const int64_t rgs = (n + CG_RG - 1) / CG_RG;
    a.cs = (int)(rgs < sms ? sms / rgs : 1);
    a.bar = sync; a.out = sync + 32; a.st = st; a.wait_ns = wait_ns;
    cudaError_t e = cudaMemsetAsync(sync, 0, 64 * sizeof(int), (cudaStream_t)s);
    if (e != cudaSuccess) return (int)e;
    const int smem = (int)(2 * n * sizeof(double));
    /* the largest of any call, as several host threads may set it */
    e = cudaFuncSetAttribute(k_dcg, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)(2 * lnb_dcg_max_n() * sizeof(double)));
    if (e != cudaSuccess) return (int)e;
    const int64_t tiles = rgs * a.cs;
    const unsigned grid = (unsigned)(tiles < sms ? tiles : sms);
    void *args[] = {&a};
    e = cudaLaunchCooperativeKernel((const void *)k_dcg, dim3(grid), dim3(CG_NT), args, (size_t)smem, (cudaStream_t)s);
    lnb_prof_count(1);
    return (int)e;
}
