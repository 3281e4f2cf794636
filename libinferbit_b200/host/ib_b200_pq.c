/*
 * ib_pq_matmul_fp32-shaped and ib_kmeans_assign-shaped entry points over the CUDA backend.
 * Host pointers in, host pointers out; the heavy arrays (PQ codes, k-means points) are copied to
 * HBM once and reused, the small ones (activations, centroids, results) move per call.
 */
#include "ib_b200_internal.h"
#include <pthread.h>
#include <sched.h>
#include <signal.h>
#include <stdatomic.h>
#include <stdlib.h>
#include <string.h>

/* ── PQ tensors cached on the device, keyed by the address of the caller's struct ── */
#define PQ_CACHE 64
typedef struct {
    const ib_b200_pq_tensor* key;
    ibcu_pq_t dev;
    void* bufs[13];
} pq_entry;
static pq_entry g_pq[PQ_CACHE];
static int g_npq;

static void pq_drop(pq_entry* e) {
    for (int i = 0; i < 13; i++) if (e->bufs[i]) ibcu_free(g_ib.ctx, e->bufs[i]);
    memset(e, 0, sizeof *e);
}
void ib_b200_pq_release(const ib_b200_pq_tensor* t) {
    ib_b200_lock();
    for (int i = 0; i < g_npq; i++)
        if (g_pq[i].key == t) { pq_drop(&g_pq[i]); g_pq[i] = g_pq[--g_npq]; memset(&g_pq[g_npq], 0, sizeof g_pq[0]); break; }
    ib_b200_unlock();
}
void ib_b200_pq_release_all(void) {
    for (int i = 0; i < g_npq; i++) pq_drop(&g_pq[i]);
    g_npq = 0;
}

static int up(void** dst, const void* src, size_t bytes) {
    int rc = ibcu_malloc(g_ib.ctx, bytes, dst);
    if (!rc) rc = ibcu_memcpy_h2d(g_ib.ctx, *dst, src, bytes);
    return rc;
}

static pq_entry* pq_get(const ib_b200_pq_tensor* t) {
    for (int i = 0; i < g_npq; i++) if (g_pq[i].key == t) return &g_pq[i];
    if (g_npq == PQ_CACHE) { ib_b200_set_error(IBCU_ERR_NOMEM, "PQ tensor cache full (%d); release some with ib_b200_pq_release", PQ_CACHE); return NULL; }
    /* what the backend takes: one or two levels (second level: at most 256 entries, one-byte or 4-bit packed indices), an
     * optional int8 outlier sidecar; anything else (uint16 second-level indices, other formats) stays with the caller */
    const int two = t->n_levels == 2;
    const int K2 = two ? (t->K_l2 > 0 ? t->K_l2 : t->K) : 0;                 /* src/pq_decode.c:1099-1101 */
    const int l2_bytes = t->l2_idx_bytes > 0 ? t->l2_idx_bytes : 1;
    if ((t->n_levels != 1 && t->n_levels != 2) || t->n_outlier < 0 || t->n_outlier >= t->N || t->G <= 0 || (t->G & 1) ||
        (t->N - t->n_outlier) % t->G || t->K < 1 || t->K > 256 || t->format < 0 || t->format > 3 ||      /* 4: the pyramid format, other arithmetic */
        !t->codebook_l1_l || !t->codebook_l1_r || !t->indices_l1_l || !t->indices_l1_r || !t->row_scale ||
        (two && (K2 > 256 || (K2 != 16 && l2_bytes != 1) || !t->codebook_l2_l || !t->codebook_l2_r || !t->indices_l2_l || !t->indices_l2_r)) ||
        (t->n_outlier > 0 && (!t->outlier_cols || !t->outlier_sidecar || !t->outlier_scale))) {
        ib_b200_set_error(IBCU_ERR_PARAM, "PQ tensor outside the supported subset (levels=%d K_l2=%d l2 index bytes=%d outliers=%d G=%d K=%d format=%d)",
                          t->n_levels, t->K_l2, t->l2_idx_bytes, t->n_outlier, t->G, t->K, t->format);
        return NULL;
    }
    pq_entry* e = &g_pq[g_npq];
    memset(e, 0, sizeof *e);
    const int C = (t->N - t->n_outlier) / t->G, half = t->G / 2;
    int rc = up(&e->bufs[0], t->codebook_l1_l, (size_t)t->K * half * 2);
    if (!rc) rc = up(&e->bufs[1], t->codebook_l1_r, (size_t)t->K * half * 2);
    if (!rc) rc = up(&e->bufs[2], t->indices_l1_l, (size_t)t->M * C);
    if (!rc) rc = up(&e->bufs[3], t->indices_l1_r, (size_t)t->M * C);
    if (!rc) rc = up(&e->bufs[4], t->row_scale, (size_t)t->M * 2);
    if (!rc && two) {
        const size_t stride = K2 == 16 ? (size_t)(C + 1) / 2 : (size_t)C;
        rc = up(&e->bufs[6], t->codebook_l2_l, (size_t)K2 * half * 2);
        if (!rc) rc = up(&e->bufs[7], t->codebook_l2_r, (size_t)K2 * half * 2);
        if (!rc) rc = up(&e->bufs[8], t->indices_l2_l, (size_t)t->M * stride);
        if (!rc) rc = up(&e->bufs[9], t->indices_l2_r, (size_t)t->M * stride);
    }
    if (!rc && t->n_outlier > 0) {
        rc = up(&e->bufs[10], t->outlier_cols, (size_t)t->n_outlier * sizeof(int32_t));
        if (!rc) rc = up(&e->bufs[11], t->outlier_sidecar, (size_t)t->M * t->n_outlier);
        if (!rc) rc = up(&e->bufs[12], t->outlier_scale, (size_t)t->n_outlier * 2);
    }
    if (!rc) {
        e->dev.M = t->M; e->dev.N = t->N; e->dev.G = t->G; e->dev.K = t->K;
        e->dev.codebook_l = e->bufs[0]; e->dev.codebook_r = e->bufs[1]; e->dev.cb_chunk_stride = 0;
        e->dev.idx_l = e->bufs[2]; e->dev.idx_r = e->bufs[3]; e->dev.row_scale = e->bufs[4];
        e->dev.K_l2 = K2; e->dev.codebook2_l = e->bufs[6]; e->dev.codebook2_r = e->bufs[7]; e->dev.idx2_l = e->bufs[8]; e->dev.idx2_r = e->bufs[9];
        e->dev.n_outlier = t->n_outlier; e->dev.outlier_cols = e->bufs[10]; e->dev.outlier_sidecar = e->bufs[11]; e->dev.outlier_scale = e->bufs[12];
        rc = ibcu_malloc(g_ib.ctx, ibcu_pq_prepared_bytes(&e->dev), &e->bufs[5]);
    }
    if (!rc) rc = ibcu_pq_prepare(g_ib.ctx, &e->dev, (uint8_t*)e->bufs[5]);
    if (!rc) rc = ibcu_sync(g_ib.ctx);
    if (ib_b200_check(rc, "PQ tensor upload")) { pq_drop(e); return NULL; }
    e->key = t;
    g_npq++;
    return e;
}

static int pq_matmul_batch_unlocked(const ib_b200_pq_tensor* t, const float* x, float* out, int B) {
    if (!t || !x || !out || B < 1) return -1;                /* src/pq_decode.c:1506 */
    if (!g_ib.ctx) { ib_b200_set_error(IBCU_ERR_STATE, "ib_b200_pq_matmul_fp32 before ib_b200_init"); return -1; }
    pq_entry* e = pq_get(t);
    if (!e) return -1;
    void *hx, *dx, *ho, *dout;
    const size_t xb = (size_t)B * t->N * sizeof(float), ob = (size_t)B * t->M * sizeof(float);
    if (ib_b200_stage(0, xb, &hx, &dx) || ib_b200_stage(2, ob, &ho, &dout)) return -1;
    memcpy(hx, x, xb);
    int rc = ibcu_memcpy_h2d(g_ib.ctx, dx, hx, xb);
    if (!rc) rc = ibcu_pq_matmul_fp32(g_ib.ctx, &e->dev, (const float*)dx, (float*)dout, B);
    if (!rc) rc = ibcu_memcpy_d2h(g_ib.ctx, ho, dout, ob);
    if (!rc) rc = ibcu_sync(g_ib.ctx);
    if (ib_b200_check(rc, "ib_b200_pq_matmul_fp32")) return -1;
    memcpy(out, ho, ob);
    return 0;
}
int ib_b200_pq_matmul_fp32_batch(const ib_b200_pq_tensor* t, const float* x, float* out, int B) {
    ib_b200_lock();
    int r = pq_matmul_batch_unlocked(t, x, out, B);
    ib_b200_unlock();
    return r;
}
int ib_b200_pq_matmul_fp32(const ib_b200_pq_tensor* t, const float* x, float* out) { return ib_b200_pq_matmul_fp32_batch(t, x, out, 1); }
int ib_b200_pq_matmul_fp32_threaded(const ib_b200_pq_tensor* t, const float* x, float* out, void* pool) {
    (void)pool;                                              /* the grid is the pool */
    return ib_b200_pq_matmul_fp32_batch(t, x, out, 1);
}
int ib_b200_pq_matmul_fp32_streaming(const ib_b200_pq_tensor* t, const float* x, float* out) { return ib_b200_pq_matmul_fp32_batch(t, x, out, 1); }

static int pq_topk_unlocked(const ib_b200_pq_tensor* t, const float* x, int K_top, float* out_logits, int32_t* out_token_ids) {
    if (!t || !x || !out_logits || !out_token_ids) return -1;            /* src/pq_decode.c:2261-2262 */
    if (K_top <= 0 || K_top > t->M) return -1;
    if (!g_ib.ctx) { ib_b200_set_error(IBCU_ERR_STATE, "ib_b200_pq_lm_head_topk before ib_b200_init"); return -1; }
    pq_entry* e = pq_get(t);
    if (!e) return -1;
    void *hx, *dx, *ho, *dout;
    const size_t xb = (size_t)t->N * sizeof(float), ob = (size_t)K_top * (sizeof(float) + sizeof(int32_t));
    if (ib_b200_stage(0, xb, &hx, &dx) || ib_b200_stage(2, ob, &ho, &dout)) return -1;
    memcpy(hx, x, xb);
    int rc = ibcu_memcpy_h2d(g_ib.ctx, dx, hx, xb);
    if (!rc) rc = ibcu_pq_lm_head_topk(g_ib.ctx, &e->dev, (const float*)dx, K_top, (float*)dout, (int32_t*)((float*)dout + K_top));
    if (!rc) rc = ibcu_memcpy_d2h(g_ib.ctx, ho, dout, ob);
    if (!rc) rc = ibcu_sync(g_ib.ctx);
    if (ib_b200_check(rc, "ib_b200_pq_lm_head_topk")) return -1;
    memcpy(out_logits, ho, (size_t)K_top * sizeof(float));
    memcpy(out_token_ids, (const float*)ho + K_top, (size_t)K_top * sizeof(int32_t));
    return 0;
}
int ib_b200_pq_lm_head_topk(const ib_b200_pq_tensor* t, const float* x, int K_top, float* out_logits, int32_t* out_token_ids) {
    ib_b200_lock();
    int r = pq_topk_unlocked(t, x, K_top, out_logits, out_token_ids);
    ib_b200_unlock();
    return r;
}

/* ── k-means ── */
/* Device arrays of a call, kept from call to call: a converter trains one codebook after another, and seven allocations
 * and frees (each waits for the device) took several milliseconds of a call whose kernels take one. What is kept is
 * bounded by KM_KEEP (larger calls give their arrays back at once), given back by ib_b200_shutdown, and used under the
 * entries' lock. */
enum { KM_X, KM_C, KM_IDX, KM_DIST, KM_SUMS, KM_COUNTS, KM_SCALARS, KM_SLOTS };
#define KM_KEEP ((size_t)256 << 20)
static struct { void* p; size_t bytes; } g_km[KM_SLOTS];

void ib_b200_kmeans_release(void) {
    for (int i = 0; i < KM_SLOTS; i++) {
        if (g_km[i].p) ibcu_free(g_ib.ctx, g_km[i].p);
        g_km[i].p = NULL; g_km[i].bytes = 0;
    }
}
static void km_trim(void) {
    size_t total = 0;
    for (int i = 0; i < KM_SLOTS; i++) total += g_km[i].bytes;
    if (total > KM_KEEP) ib_b200_kmeans_release();
}
static int km_get(int slot, size_t bytes, void** p) {
    if (g_km[slot].bytes < bytes) {
        if (g_km[slot].p) ibcu_free(g_ib.ctx, g_km[slot].p);
        g_km[slot].p = NULL; g_km[slot].bytes = 0;
        int rc = ibcu_malloc(g_ib.ctx, bytes, &g_km[slot].p);
        if (rc) { g_km[slot].p = NULL; return rc; }
        g_km[slot].bytes = bytes;
    }
    *p = g_km[slot].p;
    return 0;
}

typedef struct { void *X, *C, *idx, *dist, *sums, *counts, *inertia, *shift; } km_bufs;

/* Pageable arrays go through the pinned staging area in pieces, so that pieces are on their way while others are copied
 * (the driver's own path for pageable memory copies and transfers one after the other). One core copies 17 GB/s, a third of
 * what the bus takes, so helper threads of the call share the copying of large arrays. Starting and ending the three costs some
 * 300 us, so arrays of less than 16 MB stay with the caller. One iteration over points of 16 and 64 clusters, alone / with helpers, us: 8 MB
 * 612 / 914, 12 MB 892 / 1070, 16 MB 1168 / 823, 20 MB 1452 / 1429, 32 MB 2300 / 1571, 64 MB 5300 / 3195. CUDA calls are the
 * caller's alone. The result area is separate. */
#define KM_PIECE ((size_t)256 << 10)
#define KM_STAGE ((size_t)16 << 20)
#define KM_AREA ((int)(KM_STAGE / KM_PIECE))       /* pieces the staging area holds */
#define KM_HELPERS 3
#define KM_SHARED ((size_t)16 << 20)              /* arrays from here on are copied by several threads */

typedef struct {
    char* stage; const char* src;
    size_t bytes;
    int n;                                          /* pieces */
    atomic_int next, limit;                         /* next piece nobody has taken; pieces below limit have a free place */
    atomic_uchar* done;
} km_copy;

/* copies one piece, if there is one to take; 0: none left or no place yet */
static int km_copy_one(km_copy* c) {
    int i = atomic_load(&c->next);
    do {
        if (i >= atomic_load(&c->limit)) return 0;
    } while (!atomic_compare_exchange_weak(&c->next, &i, i + 1));
    const size_t off = (size_t)i * KM_PIECE, n = c->bytes - off < KM_PIECE ? c->bytes - off : KM_PIECE;
    memcpy(c->stage + (size_t)(i % KM_AREA) * KM_PIECE, c->src + off, n);
    atomic_store_explicit(&c->done[i], 1, memory_order_release);
    return 1;
}
static void* km_copy_helper(void* arg) {
    km_copy* c = (km_copy*)arg;
    while (atomic_load(&c->next) < c->n)
        if (!km_copy_one(c)) sched_yield();
    return NULL;
}

/* Helper threads of a copy: no more than the cores this thread may run on (a helper on the caller's core would only yield to it), and with all
 * signals blocked, so that a handler of the program never runs on one. */
static int km_helpers_start(pthread_t* helper, km_copy* c) {
    const int cores = ib_b200_cores();
    sigset_t all, caller;
    sigfillset(&all);
    if (pthread_sigmask(SIG_SETMASK, &all, &caller) != 0) return 0;
    int n = 0;
    while (n < KM_HELPERS && n + 1 < cores && pthread_create(&helper[n], NULL, km_copy_helper, c) == 0) n++;
    pthread_sigmask(SIG_SETMASK, &caller, NULL);
    return n;
}

static int km_upload(void* dst, const void* src, size_t bytes) {
    void *h, *d;
    int rc = ib_b200_stage(0, bytes < KM_STAGE ? bytes : KM_STAGE, &h, &d);
    if (rc || !bytes) return rc;
    km_copy c = { .stage = (char*)h, .src = (const char*)src, .bytes = bytes, .n = (int)((bytes + KM_PIECE - 1) / KM_PIECE) };
    atomic_init(&c.next, 0);
    atomic_init(&c.limit, c.n < KM_AREA ? c.n : KM_AREA);
    c.done = (atomic_uchar*)calloc((size_t)c.n, sizeof *c.done);
    if (!c.done) return IBCU_ERR_NOMEM;
    pthread_t helper[KM_HELPERS];
    const int helpers = bytes >= KM_SHARED ? km_helpers_start(helper, &c) : 0;
    for (int i = 0; i < c.n && !rc; i++) {
        while (!atomic_load_explicit(&c.done[i], memory_order_acquire)) km_copy_one(&c);
        const size_t off = (size_t)i * KM_PIECE, n = bytes - off < KM_PIECE ? bytes - off : KM_PIECE;
        rc = ibcu_memcpy_h2d(g_ib.ctx, (char*)dst + off, (char*)h + (size_t)(i % KM_AREA) * KM_PIECE, n);
        if (!rc && (i + 1) % KM_AREA == 0 && i + 1 < c.n) {         /* the area is used again once all of it has left */
            rc = ibcu_sync_spin(g_ib.ctx);
            atomic_store(&c.limit, c.n - i - 1 < KM_AREA ? c.n : i + 1 + KM_AREA);
        }
    }
    if (rc) atomic_store(&c.next, c.n);                              /* nothing more to take */
    for (int t = 0; t < helpers; t++) pthread_join(helper[t], NULL);
    free(c.done);
    return rc;
}

/* device arrays to host arrays; those that fit the result area together come with one wait */
typedef struct { void* dst; const void* src; size_t bytes; } km_result;
static int km_download(const km_result* r, int n) {
    size_t total = 0;
    for (int i = 0; i < n; i++) total += (r[i].bytes + 255) & ~(size_t)255;
    void *h, *d;
    int rc = ib_b200_stage(2, total < KM_STAGE ? total : KM_STAGE, &h, &d);
    if (!rc && total <= KM_STAGE) {
        size_t at = 0;
        for (int i = 0; i < n && !rc; at += (r[i].bytes + 255) & ~(size_t)255, i++) rc = ibcu_memcpy_d2h(g_ib.ctx, (char*)h + at, r[i].src, r[i].bytes);
        if (!rc) rc = ibcu_sync_spin(g_ib.ctx);
        at = 0;
        for (int i = 0; i < n && !rc; at += (r[i].bytes + 255) & ~(size_t)255, i++) memcpy(r[i].dst, (char*)h + at, r[i].bytes);
        return rc;
    }
    for (int i = 0; i < n && !rc; i++)
        for (size_t off = 0; !rc && off < r[i].bytes; off += KM_STAGE) {
            const size_t m = r[i].bytes - off < KM_STAGE ? r[i].bytes - off : KM_STAGE;
            rc = ibcu_memcpy_d2h(g_ib.ctx, h, (const char*)r[i].src + off, m);
            if (!rc) rc = ibcu_sync_spin(g_ib.ctx);
            if (!rc) memcpy((char*)r[i].dst + off, h, m);
        }
    return rc;
}

static int km_begin(km_bufs* b, const float* X, int N, int D, int K, const float* centers) {
    const size_t xb = (size_t)N * D * sizeof(float), cb = (size_t)K * D * sizeof(float);
    memset(b, 0, sizeof *b);                                       /* a step that fails leaves the rest empty */
    b->X = ib_b200_translate(X, xb);
    int rc = 0;
    if (!b->X) {
        rc = km_get(KM_X, xb, &b->X);
        if (!rc) rc = km_upload(b->X, X, xb);
    }
    if (!rc) rc = km_get(KM_C, cb, &b->C);
    if (!rc) rc = km_get(KM_IDX, (size_t)N * sizeof(int32_t), &b->idx);
    if (!rc) rc = km_get(KM_DIST, (size_t)N * sizeof(float), &b->dist);
    if (!rc) rc = km_get(KM_SUMS, cb, &b->sums);
    if (!rc) rc = km_get(KM_COUNTS, (size_t)K * sizeof(int32_t), &b->counts);
    if (!rc) rc = km_get(KM_SCALARS, 32, &b->inertia);
    if (!rc) b->shift = (char*)b->inertia + 16;
    void *h, *d;
    if (!rc) rc = ib_b200_stage(3, cb, &h, &d);                   /* not the area the points are still leaving from */
    if (!rc) { memcpy(h, centers, cb); rc = ibcu_memcpy_h2d(g_ib.ctx, b->C, h, cb); }
    return rc;
}

static int ib_b200_kmeans_assign_unlocked(const float* X, int N, int D, const float* centers, int K, int32_t* indices_out, void* pool) {
    (void)pool;
    if (!X || !centers || !indices_out || N <= 0 || K <= 0 || D <= 0) return -1;      /* src/pq_kmeans.c:403 */
    if (!g_ib.ctx) { ib_b200_set_error(IBCU_ERR_STATE, "ib_b200_kmeans_assign before ib_b200_init"); return -1; }
    km_bufs b;
    int rc = km_begin(&b, X, N, D, K, centers);
    if (!rc) rc = ibcu_kmeans_assign(g_ib.ctx, (const float*)b.X, N, D, (const float*)b.C, K, (int32_t*)b.idx, NULL);
    const km_result out = { indices_out, b.idx, (size_t)N * sizeof(int32_t) };
    if (!rc) rc = km_download(&out, 1);
    if (rc) ibcu_sync(g_ib.ctx);                                   /* nothing is left on its way out of the staging areas */
    ib_b200_check(rc, "ib_b200_kmeans_assign");
    km_trim();
    return rc ? -1 : 0;
}

/* squared length of all centroids' moves; empty clusters stay where they are */
static float km_shift(const float* now, const float* was, const int32_t* counts, int K, int D) {
    float shift = 0.0f;
    for (int k = 0; k < K; k++)
        for (int d = 0; d < D && counts[k] > 0; d++) {
            const float move = now[(size_t)k * D + d] - was[(size_t)k * D + d];
            shift += move * move;
        }
    return shift;
}

static int ib_b200_kmeans_lloyd_unlocked(const float* X, int N, int D, int K, int iters, float tol,
                         float* centers, int32_t* indices_out, double* inertia_out) {
    if (!X || !centers || N <= 0 || K <= 0 || D <= 0 || iters <= 0) return -1;
    if (!g_ib.ctx) { ib_b200_set_error(IBCU_ERR_STATE, "ib_b200_kmeans_lloyd before ib_b200_init"); return -1; }
    km_bufs b;
    int rc = km_begin(&b, X, N, D, K, centers), done = 0;
    double prev = 0.0;
    /* Whole iterations of the backend, with a tolerance as without one: both give the same bits. (With a communicator on the context
     * those would add up other ranks' tables, which this call never does.) */
    int rank = 0, world = 1;
    ibcu_comm_rank(g_ib.ctx, &rank, &world);
    const size_t KD = (size_t)K * D;
    float* was = NULL;                                             /* centroids and, behind them, those of the iteration before */
    int32_t* counts = NULL;
    const int by_tol = !(tol < 0.0f);
    if (!rc && by_tol) {
        was = (float*)malloc(2 * KD * sizeof(float) + (size_t)K * sizeof(int32_t));
        if (!was) rc = IBCU_ERR_NOMEM;
        else { counts = (int32_t*)(was + 2 * KD); memcpy(was + KD, centers, KD * sizeof(float)); }
    }
    for (int it = 0; !rc && it < iters; it++) {
        if (world == 1) {
            rc = ibcu_kmeans_lloyd_iter(g_ib.ctx, (const float*)b.X, N, D, (float*)b.C, K, (int32_t*)b.idx, (float*)b.dist,
                                        (float*)b.sums, (int32_t*)b.counts, (double*)b.inertia);
        } else {
            rc = ibcu_kmeans_assign(g_ib.ctx, (const float*)b.X, N, D, (const float*)b.C, K, (int32_t*)b.idx, (float*)b.dist);
            if (!rc) rc = ibcu_kmeans_accumulate(g_ib.ctx, (const float*)b.X, N, D, K, (const int32_t*)b.idx, (const float*)b.dist,
                                                 (float*)b.sums, (int32_t*)b.counts, (double*)b.inertia);
            if (!rc) rc = ibcu_kmeans_update(g_ib.ctx, (float*)b.C, K, D, (const float*)b.sums, (const int32_t*)b.counts, (float*)b.shift);
        }
        done = it + 1;
        if (rc || !by_tol) continue;
        /* the reference's two stopping rules (src/pq_kmeans.c:285-288); the moves are added up as it adds them (:262-282) */
        double inertia;
        const km_result now[3] = { { was, b.C, KD * sizeof(float) }, { counts, b.counts, (size_t)K * sizeof(int32_t) }, { &inertia, b.inertia, sizeof inertia } };
        rc = km_download(now, 3);
        if (rc) break;
        const float shift = km_shift(was, was + KD, counts, K, D);
        memcpy(was + KD, was, KD * sizeof(float));
        if (shift < tol) break;
        double diff = prev - inertia; if (diff < 0) diff = -diff;
        if (it > 0 && diff < (double)tol * (prev + 1e-12)) break;
        prev = inertia;
    }
    free(was);
    km_result out[3] = { { centers, b.C, (size_t)K * D * sizeof(float) } };
    int n_out = 1;
    if (indices_out) out[n_out++] = (km_result){ indices_out, b.idx, (size_t)N * sizeof(int32_t) };
    if (inertia_out) out[n_out++] = (km_result){ inertia_out, b.inertia, sizeof(double) };
    if (!rc) rc = km_download(out, n_out);
    if (rc) ibcu_sync(g_ib.ctx);
    ib_b200_check(rc, "ib_b200_kmeans_lloyd");
    km_trim();
    return rc ? -1 : done;
}

int ib_b200_kmeans_assign(const float* X, int N, int D, const float* centers, int K, int32_t* indices_out, void* pool) {
    ib_b200_lock();
    int r = ib_b200_kmeans_assign_unlocked(X, N, D, centers, K, indices_out, pool);
    ib_b200_unlock();
    return r;
}

int ib_b200_kmeans_lloyd(const float* X, int N, int D, int K, int iters, float tol,
                         float* centers, int32_t* indices_out, double* inertia_out) {
    ib_b200_lock();
    int r = ib_b200_kmeans_lloyd_unlocked(X, N, D, K, iters, tol, centers, indices_out, inertia_out);
    ib_b200_unlock();
    return r;
}
