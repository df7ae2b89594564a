// k_trsm_tiles.cu -- op(T) X = alpha B in FP64 as one persistent launch that walks
// the tile DAG.
//
// Semantics of bblas_dltrsm (bblas_trsm.h:116-202): block rows in dependency
// order, a TRSM task on each diagonal block and a GEMM task per off-diagonal
// block and column block.  Here a task produces one finished 64 x NW tile,
//     X_vs = inv(op T)_vv (alpha B_vs - sum_{u<v} op(T)_vu X_us),
// left-looking, v counting the block rows in solve order and s the column
// strips.  The inverses of the diagonal blocks come from k_trtri_blocks.
//
//   * A CTA is four tensor-core warps (DMMA) and a producer warp, which copies
//     16-deep chunks of the two operands into an mbarrier ring, waits for the
//     tiles of X they need and fetches T's part ahead of that wait; two CTAs
//     per SM.  The inverse of the diagonal block has shared memory of its own
//     and is there before the sum ends.
//   * Tasks go out by an atomic ticket, block row by block row; a strip's tiles
//     finish in order, so one counter per strip says how many are final.  A task
//     waits only on smaller tickets; every wait is bounded and reports in the
//     status word.
//   * Bound by the DMMA rate when block rows x strips fill the SMs, by the chain
//     of nb dependent tiles otherwise: 3.5 us per link with NW = 16 (flag seen 0.3,
//     X in 0.4, four chunks 1.2, right-hand side and inverse 0.4, stores and flag
//     1.1); wider strips lengthen the link and reread T less.  n = 8192 with one
//     right-hand side takes 0.45 ms per solve (0.64 as a substitution chain in one
//     CTA with two blocks of band), n = 1500 with 1500 columns 0.21 ms (0.96 as two
//     GEMM launches per block row), n = 16384 with 64 1.4 ms (3.85 as a walk of
//     64 x 64 updates with atomics); n = 8192 with 4096 columns runs at 27.6 TF/s.
#include "common.cuh"
#include "tc_sm100.cuh"

namespace lnb {
namespace tiles {

constexpr int TS = 64, NT = 128, NTHR = NT + 32;
constexpr int LDC = TS + 4;         // rows contiguous: S[k][m], ld = 4 mod 16 doubles

template <int NW> struct Cfg {
    // chunks of 16 along k; 32 for the narrow strips, whose chain feels the per-chunk cost
    static constexpr int BK = NW == 16 ? 32 : 16;
    static constexpr int ST = NW == 32 ? 4 : 3;
    static constexpr int LDR = BK + 4;             // k contiguous: S[m][k], ld = 4 mod 16 doubles
    static constexpr int ACH = TS * LDR;           // doubles of a staged chunk of op(T) (either layout)
    static_assert(BK * LDC <= ACH, "both layouts fit");
    static constexpr int STAGE = ACH + NW * LDR;
    static constexpr int RING = ST * STAGE;
    static_assert(NW * LDC <= RING, "the right-hand side of the diagonal product reuses the ring");
    static constexpr int SMEM = (RING + TS * LDC) * (int)sizeof(double);
};

struct Args {
    const double *T; int64_t ldt;
    const double *dinv;             // 64 x 64 inverses of the diagonal blocks of T, column-major
    double *B; int64_t ldb;
    int64_t n, nrhs;
    double alpha;
    int nb, ns, fwd;
    int64_t ntasks;
    int *ticket, *prog;             // prog[s]: tiles of strip s that are final
    int ticket0;                    // first ticket handed out (0; 1 only in the wait self-test)
    lnb_status_t *st;
    long long wait_ns;
};

struct Shared {
    uint64_t full[4], empty[4], dfull;
    int task, abort;
};

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
// spin until *f >= target and return it; -1 after wait_ns or a recorded timeout
LNB_DEV int wait_prog(const int *f, int target, const Args &a)
{
    const uint64_t t0 = globaltimer();
    for (int it = 0;; ++it) {
        const int v = ld_acquire(f);
        if (v >= target) return v;
        if ((it & 15) == 15) {
            if (ld_acquire(&a.st->timeout) != 0) return -1;
            if ((long long)(globaltimer() - t0) > a.wait_ns) return -1;
        }
        if (it > 8) __nanosleep(40);
    }
}
LNB_DEV void give_up(const Args &a, int site, int item)
{
    if (atomicCAS(&a.st->timeout, 0, site) == 0) a.st->timeout_item = item;
}
LNB_DEV void arrive_copied(uint64_t *bar)
{
    asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}
LNB_DEV void cp16(uint32_t d, const double *g, int bytes)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(d), "l"(g), "r"(bytes));
}
LNB_DEV void cp8(uint32_t d, const double *g, int bytes)
{
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(d), "l"(g), "r"(bytes));
}

// NC columns of 64 contiguous elements: dst[c * LDC + r] = X[r + c ld], zero where
// r >= nr or c >= nc; by the producer warp.  Pointers step from column to column:
// the warp issues alone, and its address arithmetic is the chunk's latency.
template <int NC>
LNB_DEV void load64(double *dst, const double *X, int64_t ld, int nr, int nc, bool vec, int lane)
{
    if (vec) {
        const int r = 2 * lane, bytes = r + 1 < nr ? 16 : r < nr ? 8 : 0;
        uint32_t d = smem_u32(dst + r);
        const double *g = X + (bytes ? r : 0);
        if (nc >= NC) {
#pragma unroll
            for (int c = 0; c < NC; ++c, g += ld) cp16(d + c * (LDC * 8), g, bytes);
        } else {
#pragma unroll 1
            for (int c = 0; c < NC; ++c, d += LDC * 8) cp16(d, c < nc ? g + c * ld : X, c < nc ? bytes : 0);
        }
    } else {
        const int b0 = lane < nr ? 8 : 0, b1 = lane + 32 < nr ? 8 : 0;
        uint32_t d = smem_u32(dst + lane);
        const double *g0 = X + (b0 ? lane : 0), *g1 = X + (b1 ? lane + 32 : 0);
#pragma unroll 4
        for (int c = 0; c < NC; ++c, d += LDC * 8) {
            const bool in = c < nc;
            cp8(d, in ? g0 : X, in ? b0 : 0);
            cp8(d + 256, in ? g1 : X, in ? b1 : 0);
            g0 += ld;
            g1 += ld;
        }
    }
}
// NC columns of RUN (16 or 32) contiguous elements: dst[c * (RUN + 4) + r] = X[r + c ld]
template <int RUN, int NC>
LNB_DEV void load_run(double *dst, const double *X, int64_t ld, int nr, int nc, bool vec, int lane)
{
    constexpr int LDR = RUN + 4, CV = 64 / RUN, CE = 32 / RUN;     // columns per instruction
    if (vec) {
        const int r = 2 * (lane & (RUN / 2 - 1)), bytes = r + 1 < nr ? 16 : r < nr ? 8 : 0;
        int c = lane / (RUN / 2);
        uint32_t d = smem_u32(dst + c * LDR + r);
        const double *g = X + (bytes ? r : 0) + c * ld;
        const int64_t step = CV * ld;
        if (nc >= NC) {
#pragma unroll
            for (int it = 0; it < NC / CV; ++it, g += step) cp16(d + it * (CV * LDR * 8), g, bytes);
        } else {
#pragma unroll 1
            for (int it = 0; it < NC / CV; ++it, c += CV, d += CV * LDR * 8, g += step)
                cp16(d, c < nc ? g : X, c < nc ? bytes : 0);
        }
    } else {
        const int r = lane & (RUN - 1), bytes = r < nr ? 8 : 0;
        int c = lane / RUN;
        uint32_t d = smem_u32(dst + c * LDR + r);
        const double *g = X + (bytes ? r : 0) + c * ld;
        const int64_t step = CE * ld;
#pragma unroll 4
        for (int it = 0; it < NC / CE; ++it, c += CE, d += CE * LDR * 8, g += step) cp8(d, c < nc ? g : X, c < nc ? bytes : 0);
    }
}

LNB_DEV int blk_len(const Args &a, int64_t o) { return (int)(a.n - o < TS ? a.n - o : TS); }

// the producer's side of task (v, s); q counts the chunks of all tasks
template <int NW, bool TR>
LNB_DEV bool produce(const Args &a, int v, int s, double *sm, Shared &sh, int &q)
{
    using C = Cfg<NW>;
    constexpr int BK = C::BK;
    const int lane = threadIdx.x & 31;
    const bool vt = ((uintptr_t)a.T % 16 == 0) && a.ldt % 2 == 0;
    const bool vb = ((uintptr_t)a.B % 16 == 0) && a.ldb % 2 == 0;
    const int64_t oi = (int64_t)(a.fwd ? v : a.nb - 1 - v) * TS;
    const int64_t c0 = (int64_t)s * NW;
    const int rows = blk_len(a, oi), cols = (int)(a.nrhs - c0 < NW ? a.nrhs - c0 : NW);
    const double *D = a.dinv + oi * TS;
    load64<TS>(sm + C::RING, D, TS, TS, TS, true, lane);
    arrive_copied(&sh.dfull);
    int known = 0;
    bool ok = true;
    constexpr int CPT = TS / BK;                     // chunks per tile
    for (int u = 0; u < v && ok; ++u) {
        const int64_t oj = (int64_t)(a.fwd ? u : a.nb - 1 - u) * TS;     // block u in solve order
        const int kt = blk_len(a, oj);
        // op(T)(m, k) = T[oi + m + (oj + k) ldt], or T[oj + k + (oi + m) ldt]
        const double *Tu = a.T + (TR ? oj + oi * a.ldt : oi + oj * a.ldt);
        const double *Bu = a.B + oj + c0 * a.ldb;
        auto load_t = [&](int c) {                   // chunk c of the tile, into the slot of chunk q + c
            const int qc = q + c, st = qc % C::ST;
            if (qc >= C::ST && !bar_wait(&sh.empty[st], ((qc / C::ST) - 1) & 1, 4 * a.wait_ns, sh)) ok = false;
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) return;
            const int kn = kt - c * BK < 0 ? 0 : kt - c * BK < BK ? kt - c * BK : BK;
            double *as = sm + st * C::STAGE;
            if (!TR) load64<BK>(as, kn ? Tu + c * BK * a.ldt : a.T, a.ldt, rows, kn, vt, lane);
            else load_run<BK, TS>(as, kn ? Tu + c * BK : a.T, a.ldt, kn, rows, vt, lane);
        };
        auto load_b = [&](int c) {
            const int st = (q + c) % C::ST;
            const int kn = kt - c * BK < 0 ? 0 : kt - c * BK < BK ? kt - c * BK : BK;
            load_run<BK, NW>(sm + st * C::STAGE + C::ACH, kn ? Bu + c * BK : a.B, a.ldb, kn, cols, vb, lane);
            arrive_copied(&sh.full[st]);
        };
        int ahead = 0;                               // chunks whose part of T goes out before the wait
        if (u >= known) {
            constexpr int AH = C::ST < CPT ? C::ST : CPT;
            for (; ahead < AH && ok; ++ahead) load_t(ahead);
            if (!ok) break;
            if (lane == 0) known = wait_prog(a.prog + s, u + 1, a);
            known = __shfl_sync(0xffffffffu, known, 0);
            if (known < 0) {
                ok = false;
                break;
            }
        }
        for (int c = 0; c < CPT && ok; ++c) {
            if (c >= ahead) load_t(c);
            if (ok) load_b(c);
        }
        q += CPT;
    }
    if (!ok) {
        if (lane == 0) {
            give_up(a, 51, v * a.ns + s);
            sh.abort = 1;
        }
        cp_async_wait<0>();
    }
    return ok;
}

// the multiplying warps' side
template <int NW, bool TR>
LNB_DEV bool multiply(const Args &a, int v, int s, double *sm, Shared &sh, int &q, int &nd)
{
    using C = Cfg<NW>;
    constexpr int BK = C::BK, LDR = C::LDR;
    constexpr int WN = NW == 64 ? 2 : 1, WM = 4 / WN;       // warp grid of the sum
    constexpr int MI = TS / WM / 16, NI = NW / WN / 8;
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5, g = lane >> 2, t = lane & 3;
    const int wm = w / WN, wn = w % WN;
    const int64_t oi = (int64_t)(a.fwd ? v : a.nb - 1 - v) * TS, c0 = (int64_t)s * NW;
    const int rows = blk_len(a, oi), cols = (int)(a.nrhs - c0 < NW ? a.nrhs - c0 : NW);
    double *Rs = sm, *Ds = sm + C::RING, *Bt = a.B + oi + c0 * a.ldb;
    // the sum over a tile's 64 terms, and over the tiles: one accumulator through up
    // to n terms doubled the error of a solve with n = 8192
    double acc[MI][NI][4], tot[MI][NI][4];
#pragma unroll
    for (int mi = 0; mi < MI; ++mi)
#pragma unroll
        for (int ni = 0; ni < NI; ++ni)
#pragma unroll
            for (int e = 0; e < 4; ++e) acc[mi][ni][e] = tot[mi][ni][e] = 0.0;
    // B's own entries are fetched ahead of the last 64 terms and used after them
    double rhs[MI][NI][4];
    auto take_rhs = [&]() {
#pragma unroll
        for (int mi = 0; mi < MI; ++mi)
#pragma unroll
            for (int ni = 0; ni < NI; ++ni)
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const int r = wm * (TS / WM) + mi * 16 + g + ((e & 2) ? 8 : 0);
                    const int c = wn * (NW / WN) + ni * 8 + 2 * t + (e & 1);
                    rhs[mi][ni][e] = r < rows && c < cols ? __ldcg(Bt + r + c * a.ldb) : 0.0;
                }
    };
    bool ok = true;
    const int nch = v * (TS / BK);
    // (64 columns: at the end, the registers hold the sums)
    if (nch == 0 && NW < 64) take_rhs();
    for (int c = 0; c < nch; ++c) {
        if (NW < 64 && c == nch - TS / BK) take_rhs();
        const int st = q % C::ST;
        if (!bar_wait(&sh.full[st], (q / C::ST) & 1, 4 * a.wait_ns, sh)) {
            ok = false;
            break;
        }
        const double *as = sm + st * C::STAGE, *bs = as + C::ACH + (wn * (NW / WN) + g) * LDR + t;
#pragma unroll
        for (int kq = 0; kq < BK / 4; ++kq) {
            double a0[MI], a1[MI], b0[NI];
#pragma unroll
            for (int mi = 0; mi < MI; ++mi) {
                const int r = wm * (TS / WM) + mi * 16 + g;
                a0[mi] = TR ? as[r * LDR + kq * 4 + t] : as[(kq * 4 + t) * LDC + r];
                a1[mi] = TR ? as[(r + 8) * LDR + kq * 4 + t] : as[(kq * 4 + t) * LDC + r + 8];
            }
#pragma unroll
            for (int ni = 0; ni < NI; ++ni) b0[ni] = bs[ni * 8 * LDR + kq * 4];
#pragma unroll
            for (int mi = 0; mi < MI; ++mi)
#pragma unroll
                for (int ni = 0; ni < NI; ++ni) dmma16x8x4(acc[mi][ni], a0[mi], a1[mi], b0[ni]);
        }
        __syncwarp();
        if (lane == 0) tc::mbar_arrive(&sh.empty[st]);
        ++q;
        if (c % (TS / BK) == TS / BK - 1) {
#pragma unroll
            for (int mi = 0; mi < MI; ++mi)
#pragma unroll
                for (int ni = 0; ni < NI; ++ni)
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        tot[mi][ni][e] += acc[mi][ni][e];
                        acc[mi][ni][e] = 0.0;
                    }
        }
    }
    if (!mma_sync_and(ok)) return false;             // the ring is free
    if (NW == 64) take_rhs();
#pragma unroll
    for (int mi = 0; mi < MI; ++mi)
#pragma unroll
        for (int ni = 0; ni < NI; ++ni)
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int r = wm * (TS / WM) + mi * 16 + g + ((e & 2) ? 8 : 0);
                const int c = wn * (NW / WN) + ni * 8 + 2 * t + (e & 1);
                Rs[c * LDC + r] = fma(a.alpha, rhs[mi][ni][e], -tot[mi][ni][e]);
            }
    ok = bar_wait(&sh.dfull, nd & 1, 4 * a.wait_ns, sh);
    ++nd;
    if (!mma_sync_and(ok)) return false;
    // X = inv(op T)_vv R: 16 rows per warp; the inverse is triangular, lower in solve order
    double o[NW / 8][4];
#pragma unroll
    for (int ni = 0; ni < NW / 8; ++ni)
#pragma unroll
        for (int e = 0; e < 4; ++e) o[ni][e] = 0.0;
    const int kb = a.fwd ? 0 : 4 * w, ke = a.fwd ? 4 * w + 4 : TS / 4;
    for (int kq = kb; kq < ke; ++kq) {
        const int m = 16 * w + g, k = 4 * kq + t;
        const double a0 = TR ? Ds[m * LDC + k] : Ds[k * LDC + m], a1 = TR ? Ds[(m + 8) * LDC + k] : Ds[k * LDC + m + 8];
#pragma unroll
        for (int ni = 0; ni < NW / 8; ++ni) dmma16x8x4(o[ni], a0, a1, Rs[(8 * ni + g) * LDC + k]);
    }
#pragma unroll
    for (int ni = 0; ni < NW / 8; ++ni)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int r = 16 * w + g + ((e & 2) ? 8 : 0), c = 8 * ni + 2 * t + (e & 1);
            if (r < rows && c < cols) Bt[r + c * a.ldb] = o[ni][e];
        }
    mma_sync();
    if (tid == 0) {
        __threadfence();
        asm volatile("st.relaxed.gpu.global.s32 [%0], %1;" ::"l"(a.prog + s), "r"(v + 1) : "memory");
    }
    return true;
}

template <int NW, bool TR>
__global__ void __launch_bounds__(NTHR, 2) k_trsm_tiles(Args a)
{
    using C = Cfg<NW>;
    extern __shared__ __align__(128) double sm[];
    __shared__ __align__(8) Shared sh;
    const int warp = threadIdx.x >> 5;
    if (threadIdx.x == 0) {
        for (int s = 0; s < C::ST; ++s) {
            tc::mbar_init(&sh.full[s], 32);
            tc::mbar_init(&sh.empty[s], NT / 32);
        }
        tc::mbar_init(&sh.dfull, 32);
        sh.abort = 0;
        tc::fence_mbar_init();
    }
    int q = 0, nd = 0;
    for (;;) {
        __syncthreads();
        if (*(volatile int *)&sh.abort) break;       // the same for every thread: set before the barrier
        if (threadIdx.x == 0) sh.task = atomicAdd(a.ticket, 1) + a.ticket0;
        __syncthreads();
        const int tk = sh.task;
        if (tk >= a.ntasks) break;
        const int v = tk / a.ns, s = tk - v * a.ns;
        if (warp == NT / 32 ? !produce<NW, TR>(a, v, s, sm, sh, q) : !multiply<NW, TR>(a, v, s, sm, sh, q, nd)) {
            if (threadIdx.x == 0) give_up(a, 52, v * a.ns + s);   // stands unless the producer's own wait ran out
            sh.abort = 1;
        }
    }
    cp_async_wait<0>();                              // what the producer issued for a task that gave up
}

template <int NW>
static int launch(const Args &a, bool tr, int sms, lnb_stream_t s)
{
    const auto kernel = tr ? k_trsm_tiles<NW, true> : k_trsm_tiles<NW, false>;
    const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg<NW>::SMEM);
    if (e != cudaSuccess) return (int)e;
    const int64_t grid = a.ntasks < 2 * sms ? a.ntasks : 2 * sms;
    kernel<<<(unsigned)grid, NTHR, Cfg<NW>::SMEM, (cudaStream_t)s>>>(a);
    lnb_prof_count(1);
    return (int)cudaGetLastError();
}

}  // namespace tiles
}  // namespace lnb

// strips of at least 16 columns: one counter each, and the ticket
extern "C" int64_t lnb_trsm_tiles_ints(int64_t nrhs) { return 32 + (nrhs + 15) / 16; }

// op(T) X = alpha B, T n x n (uplo as stored), B n x nrhs in place; dinv: the 64 x 64
// inverses of T's diagonal blocks; sync: lnb_trsm_tiles_ints(nrhs) ints (zeroed here)
extern "C" int lnb_k_trsm_tiles_f64(char uplo, char trans, int64_t n, int64_t nrhs, double alpha, const double *T,
                                    int64_t ldt, const double *dinv, double *B, int64_t ldb, int *sync,
                                    lnb_status_t *st, long long wait_ns, int sms, int ticket0, lnb_stream_t s)
{
    using namespace lnb::tiles;
    if (n <= 0 || nrhs <= 0) return 0;
    const int64_t nb = (n + TS - 1) / TS;
    // Strip width by the size of B.  Measured (us, NW = 16 / 32 / 64):  n = 1500: 128
    // columns 170 / 191 / 252, 256 176 / 198 / 252, 1500 - / 246 / 284;  n = 4096: 128
    // 370 / 432 / 584, 256 494 / 467 / 650;  n = 16384: 32 1291 / 1570 / 2339, 64 1766 /
    // 1703 / 2396;  n = 3000, 3000 columns 1253 (32) / 1179 (64);  5000, 5000 5400 / 4860.
    const int64_t work = n * nrhs;
    const int nw = work <= (1 << 19) ? 16 : work <= (1 << 22) ? 32 : 64;
    Args a;
    a.T = T; a.ldt = ldt; a.dinv = dinv; a.B = B; a.ldb = ldb; a.n = n; a.nrhs = nrhs; a.alpha = alpha;
    a.nb = (int)nb; a.ns = (int)((nrhs + nw - 1) / nw); a.fwd = (uplo == 'L') == (trans == 'N');
    a.ntasks = nb * a.ns;
    if (a.ntasks > INT32_MAX - 1024) return (int)cudaErrorInvalidValue;
    a.ticket = sync; a.ticket0 = ticket0; a.prog = sync + 32; a.st = st; a.wait_ns = wait_ns;
    const cudaError_t e = cudaMemsetAsync(sync, 0, (size_t)lnb_trsm_tiles_ints(nrhs) * sizeof(int), (cudaStream_t)s);
    if (e != cudaSuccess) return (int)e;
    const bool tr = trans == 'T';
    return nw == 64 ? launch<64>(a, tr, sms, s) : nw == 32 ? launch<32>(a, tr, sms, s) : launch<16>(a, tr, sms, s);
}
