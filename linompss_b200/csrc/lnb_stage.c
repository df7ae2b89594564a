/*
 * lnb_stage.c -- copies between pageable host matrices and the device (host C).
 *
 * cudaMemcpy2DAsync from or to pageable memory goes through the driver's own
 * bounce buffer on the calling thread: 10 - 18 GB/s, where the link moves 50.
 * Large copies here go through pinned buffers of the context instead: a few
 * threads take chunks of whole columns in turn, copy each between the caller's
 * matrix and a pinned slot, and issue the slot's device copy, so the host copies
 * run in parallel and beside the link.  18 MB (the lower triangle of n = 2048)
 * takes 0.85 ms instead of 1.6 (a host call at n = 2048: 3.9 -> 2.5 ms).
 *
 * The threads live for one call; the pinned slots (LNB_STAGE_SLOTS MB) stay with
 * the context until lnb_release_workspace.  A mutex serializes the
 * calls of several host threads.  Small copies, and copies of memory that is
 * pinned, managed or on a device, take the driver's path as before.
 */
#include <cuda.h>
#include <pthread.h>
#include <stdatomic.h>
#include <string.h>
#include <unistd.h>

#include "lnb_host.h"

#define STAGE_CHUNK ((size_t)1 << 20)
/* measured on 16 cores: below 4 MB the threads cost what they save */
#define STAGE_MIN ((size_t)4 << 20)
#define STAGE_THREADS 4       /* 4 to 10 measure the same */
_Static_assert(LNB_STAGE_SLOTS == 2 * STAGE_THREADS, "two slots per thread");

typedef struct {
    lnb_ctx *c;
    const lnb_rect *r;
    int nr, to_device;
    size_t dpitch, hpitch;
    cudaStream_t s;
    atomic_long next;           /* the next column, counted through all rectangles in chunks */
    atomic_int err;
    CUcontext ctx;              /* the caller's: the streams and events belong to it */
    CUresult (*set_current)(CUcontext);
} stage_job;

typedef struct {
    stage_job *j;
    int w;                      /* thread: slots 2w and 2w + 1 */
    pthread_t th;
} stage_worker;

static pthread_mutex_t g_stage_lock = PTHREAD_MUTEX_INITIALIZER;

/* columns of rectangle r per chunk */
static size_t chunk_cols(const lnb_rect *r)
{
    const size_t k = STAGE_CHUNK / (r->width ? r->width : 1);
    return k ? k : 1;
}

/* the chunk with number k; 0 past the last one */
static int find_chunk(const stage_job *j, long k, const lnb_rect **r, size_t *col, size_t *ncol)
{
    for (int i = 0; i < j->nr; ++i) {
        const size_t cc = chunk_cols(&j->r[i]);
        const long n = (long)((j->r[i].cols + cc - 1) / cc);
        if (k < n) {
            *r = &j->r[i];
            *col = (size_t)k * cc;
            *ncol = j->r[i].cols - *col < cc ? j->r[i].cols - *col : cc;
            return 1;
        }
        k -= n;
    }
    return 0;
}

static void pack(const stage_job *j, char *slot, const lnb_rect *r, size_t col, size_t ncol, int in)
{
    char *h = r->host + col * j->hpitch;
    for (size_t q = 0; q < ncol; ++q) {
        if (in) memcpy(slot + q * r->width, h + q * j->hpitch, r->width);
        else memcpy(h + q * j->hpitch, slot + q * r->width, r->width);
    }
}

static void *stage_run(void *arg)
{
    stage_worker *me = (stage_worker *)arg;
    stage_job *j = me->j;
    lnb_ctx *c = j->c;
    const lnb_rect *r[2] = {NULL, NULL};
    size_t col[2] = {0, 0}, ncol[2] = {0, 0};
    /* The started threads join the caller's context, which need not be the device's primary
     * one (cudaSetDevice would make that current); the caller's own thread has it. */
    int e = me->w && j->set_current(j->ctx) != CUDA_SUCCESS ? (int)cudaErrorInvalidResourceHandle : 0;
    for (int k = 0; !e; k ^= 1) {
        const int slot = 2 * me->w + k;
        char *buf = (char *)c->stage + (size_t)slot * STAGE_CHUNK;
        if (r[k]) {                                    /* the slot's copy of two chunks ago */
            if ((e = (int)cudaEventSynchronize(c->stage_ev[slot]))) break;
            if (!j->to_device) pack(j, buf, r[k], col[k], ncol[k], 0);
            r[k] = NULL;
        }
        if (!find_chunk(j, atomic_fetch_add(&j->next, 1), &r[k], &col[k], &ncol[k])) break;
        char *d = r[k]->dev + col[k] * j->dpitch;
        const size_t w = r[k]->width;
        if (j->to_device) {
            pack(j, buf, r[k], col[k], ncol[k], 1);
            e = (int)cudaMemcpy2DAsync(d, j->dpitch, buf, w, w, ncol[k], cudaMemcpyHostToDevice, j->s);
        } else {
            e = (int)cudaMemcpy2DAsync(buf, w, d, j->dpitch, w, ncol[k], cudaMemcpyDeviceToHost, j->s);
        }
        if (!e) e = (int)cudaEventRecord(c->stage_ev[slot], j->s);
    }
    /* what is still in flight: the slots are free again when this returns */
    for (int k = 0; k < 2; ++k)
        if (r[k]) {
            const int e2 = (int)cudaEventSynchronize(c->stage_ev[2 * me->w + k]);
            if (!e) e = e2;
            if (!j->to_device && !e) pack(j, (char *)c->stage + (size_t)(2 * me->w + k) * STAGE_CHUNK, r[k], col[k], ncol[k], 0);
        }
    if (e) atomic_store(&j->err, e);
    return NULL;
}

/* the driver's functions for the current context of a thread; 0 if they cannot be had */
static int context_calls(CUcontext *now, CUresult (**set_current)(CUcontext))
{
    void *get = NULL, *set = NULL;
    enum cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuCtxGetCurrent", &get, cudaEnableDefault, &q) != cudaSuccess || !get ||
        cudaGetDriverEntryPoint("cuCtxSetCurrent", &set, cudaEnableDefault, &q) != cudaSuccess || !set) {
        cudaGetLastError();
        return 0;
    }
    *set_current = (CUresult (*)(CUcontext))set;
    return ((CUresult (*)(CUcontext *))get)(now) == CUDA_SUCCESS;
}

static int is_pageable(const void *p)
{
    struct cudaPointerAttributes a;
    if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
        cudaGetLastError();
        return 1;
    }
    return a.type == cudaMemoryTypeUnregistered;
}

static int stage_ready(lnb_ctx *c)
{
    if (c->stage) return 1;
    for (int i = 0; i < LNB_STAGE_SLOTS; ++i)
        if (!c->stage_ev[i] && cudaEventCreateWithFlags(&c->stage_ev[i], cudaEventDisableTiming) != cudaSuccess) {
            cudaGetLastError();
            c->stage_ev[i] = NULL;
            return 0;
        }
    if (cudaMallocHost(&c->stage, LNB_STAGE_SLOTS * STAGE_CHUNK) != cudaSuccess) {
        cudaGetLastError();
        c->stage = NULL;
        return 0;
    }
    return 1;
}

int lnb_copy_rects(lnb_ctx *c, const lnb_rect *r, int nr, size_t dpitch, size_t hpitch, int to_device,
                   cudaStream_t s, const char *where)
{
    size_t total = 0, widest = 0;
    for (int i = 0; i < nr; ++i) {
        total += r[i].width * r[i].cols;
        if (r[i].width > widest) widest = r[i].width;
    }
    const long cpus = sysconf(_SC_NPROCESSORS_ONLN);
    if (total >= STAGE_MIN && widest <= STAGE_CHUNK && cpus > 2 && is_pageable(r[0].host)) {
        pthread_mutex_lock(&g_stage_lock);
        if (stage_ready(c)) {
            stage_job j = {.c = c, .r = r, .nr = nr, .to_device = to_device, .dpitch = dpitch, .hpitch = hpitch, .s = s};
            stage_worker w[STAGE_THREADS];
            int nt = cpus - 1 < STAGE_THREADS ? (int)cpus - 1 : STAGE_THREADS, started = 1;
            if (!context_calls(&j.ctx, &j.set_current)) nt = 1;
            atomic_init(&j.next, 0);
            atomic_init(&j.err, 0);
            for (int i = 0; i < nt; ++i) {
                w[i].j = &j;
                w[i].w = i;
            }
            /* a thread that cannot be started leaves its share to the others */
            for (; started < nt; ++started)
                if (pthread_create(&w[started].th, NULL, stage_run, &w[started])) break;
            stage_run(&w[0]);
            for (int i = 1; i < started; ++i) pthread_join(w[i].th, NULL);
            pthread_mutex_unlock(&g_stage_lock);
            const int e = atomic_load(&j.err);
            return e ? lnb_cuda_error(e, where) : 0;
        }
        pthread_mutex_unlock(&g_stage_lock);
    }
    for (int i = 0; i < nr; ++i) {
        if (!r[i].width || !r[i].cols) continue;
        const int e = to_device ? (int)cudaMemcpy2DAsync(r[i].dev, dpitch, r[i].host, hpitch, r[i].width, r[i].cols,
                                                         cudaMemcpyHostToDevice, s)
                                : (int)cudaMemcpy2DAsync(r[i].host, hpitch, r[i].dev, dpitch, r[i].width, r[i].cols,
                                                         cudaMemcpyDeviceToHost, s);
        if (e) return lnb_cuda_error(e, where);
    }
    return 0;
}

int lnb_copy_matrix(lnb_ctx *c, void *dev, size_t dpitch, const void *host, size_t hpitch, size_t width, size_t cols,
                    int to_device, cudaStream_t s, const char *where)
{
    const lnb_rect r = {(char *)dev, (char *)host, width, cols};
    return lnb_copy_rects(c, &r, 1, dpitch, hpitch, to_device, s, where);
}

int lnb_copy_lower_f64(lnb_ctx *c, double *dev, int64_t ldd, const double *host, int64_t ldh, int64_t n, int64_t step,
                       int to_device, cudaStream_t s)
{
    enum { NR = 64 };
    lnb_rect r[NR];
    for (int64_t c0 = 0; c0 < n;) {
        int k = 0;
        for (; k < NR && c0 < n; ++k, c0 += step) {
            r[k].dev = (char *)(dev + c0 + c0 * ldd);
            r[k].host = (char *)(host + c0 + c0 * ldh);
            r[k].width = (size_t)(n - c0) * sizeof(double);
            r[k].cols = (size_t)(n - c0 < step ? n - c0 : step);
        }
        const int e = lnb_copy_rects(c, r, k, (size_t)ldd * sizeof(double), (size_t)ldh * sizeof(double), to_device, s,
                                     "lower block columns");
        if (e) return e;
    }
    return 0;
}

void lnb_stage_release(lnb_ctx *c)
{
    pthread_mutex_lock(&g_stage_lock);
    if (c->stage) cudaFreeHost(c->stage);
    c->stage = NULL;
    pthread_mutex_unlock(&g_stage_lock);
}
