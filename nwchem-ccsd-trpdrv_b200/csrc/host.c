/*
 * C host layer of libtrpdrv_b200.so: argument validation, device context, plans (device storage,
 * work queues, CUDA-graph capture of the fused launch sequence), and the reference's drop-in entry
 * points.  All device work is enqueued through the extern "C" launchers of launch.h.
 */
#include "trpdrv.h"
#include "launch.h"
#include "stage.h"

#include <cuda_runtime_api.h>
#include <fcntl.h>
#include <math.h>
#include <pthread.h>
#include <stdarg.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>
#include <sys/file.h>
#include <unistd.h>

int trpdrv_plain_init(void);

/* ------------------------------------------------------------------------------------------ */
/* errors                                                                                       */
/* ------------------------------------------------------------------------------------------ */

static _Thread_local int t_status = TRPDRV_OK;
static _Thread_local char t_message[512];

static int fail(int status, const char *fmt, ...)
{
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(t_message, sizeof t_message, fmt, ap);
    va_end(ap);
    t_status = status;
    return status;
}

/* Records a failure from another translation unit (declared in launch.h). */
int trpdrv_record_error(int status, const char *message)
{
    return fail(status, "%s", message ? message : "");
}

int trpdrv_last_error(void) { return t_status; }
const char *trpdrv_last_error_message(void) { return t_message; }
void trpdrv_clear_error(void)
{
    t_status = TRPDRV_OK;
    t_message[0] = '\0';
}

const char *trpdrv_status_string(int status)
{
    switch (status) {
    case TRPDRV_OK: return "ok";
    case TRPDRV_ERR_ARG: return "invalid argument";
    case TRPDRV_ERR_CUDA: return "CUDA runtime error";
    case TRPDRV_ERR_NOMEM: return "out of memory";
    case TRPDRV_ERR_NODEV: return "no usable sm_100 device";
    case TRPDRV_ERR_STATE: return "call out of order";
    case TRPDRV_ERR_UNSUPPORTED: return "unsupported";
    case TRPDRV_ERR_DEVICE: return "device-side check failed";
    default: return "unknown status";
    }
}

#define CUDA_TRY(call)                                                                              \
    do {                                                                                            \
        cudaError_t e_ = (call);                                                                    \
        if (e_ != cudaSuccess) {                                                                    \
            cudaGetLastError(); /* reported here: the next launch's check must not find it again */ \
            return fail(e_ == cudaErrorMemoryAllocation ? TRPDRV_ERR_NOMEM : TRPDRV_ERR_CUDA,       \
                        "%s: %s (%s:%d)", #call, cudaGetErrorString(e_), __FILE__, __LINE__);       \
        }                                                                                           \
    } while (0)

#define LAUNCH_TRY(call)                                                                            \
    do {                                                                                            \
        int e_ = (call);                                                                            \
        if (e_ != 0)                                                                                \
            return fail(TRPDRV_ERR_CUDA, "%s: %s (%s:%d)", #call, cudaGetErrorString((cudaError_t)e_), \
                        __FILE__, __LINE__);                                                        \
    } while (0)

#define TRY(call)                                                                                   \
    do {                                                                                            \
        int s_ = (call);                                                                            \
        if (s_ != TRPDRV_OK) return s_;                                                             \
    } while (0)

/* ------------------------------------------------------------------------------------------ */
/* device                                                                                       */
/* ------------------------------------------------------------------------------------------ */

#define TRPDRV_MAX_DEVICES 64
static pthread_mutex_t g_init_mu = PTHREAD_MUTEX_INITIALIZER;
static int g_init_done[TRPDRV_MAX_DEVICES];

/* Selects `device` (-1 = current), checks that it is an sm_100 part, and sets the kernels'
 * shared-memory limits once per device. */
static int ensure_device(int device, int *out_dev, int *out_nsm)
{
    int count = 0;
    cudaError_t e = cudaGetDeviceCount(&count);
    if (e != cudaSuccess || count == 0)
        return fail(TRPDRV_ERR_NODEV, "no CUDA device available (%s)", cudaGetErrorString(e));
    int dev = device;
    if (dev < 0) CUDA_TRY(cudaGetDevice(&dev));
    if (dev >= count || dev >= TRPDRV_MAX_DEVICES) return fail(TRPDRV_ERR_ARG, "device %d out of range", dev);
    CUDA_TRY(cudaSetDevice(dev));
    int major = 0, minor = 0, nsm = 0;
    CUDA_TRY(cudaDeviceGetAttribute(&major, cudaDevAttrComputeCapabilityMajor, dev));
    CUDA_TRY(cudaDeviceGetAttribute(&minor, cudaDevAttrComputeCapabilityMinor, dev));
    CUDA_TRY(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
    if (major != 10 || minor != 0)
        return fail(TRPDRV_ERR_NODEV, "device %d is sm_%d%d; libtrpdrv_b200 is built for sm_100a only", dev,
                    major, minor);
    pthread_mutex_lock(&g_init_mu);
    int rc = 0;
    if (!g_init_done[dev]) {
        rc = trpdrv_fused_tma_init();
        if (!rc) rc = trpdrv_plain_init();
        if (!rc) rc = trpdrv_oz_init();
        if (!rc) g_init_done[dev] = 1;
    }
    pthread_mutex_unlock(&g_init_mu);
    if (rc) return fail(TRPDRV_ERR_CUDA, "kernel attribute setup failed: %s", cudaGetErrorString((cudaError_t)rc));
    if (out_dev) *out_dev = dev;
    if (out_nsm) *out_nsm = nsm;
    return TRPDRV_OK;
}

static int check_shape(const trpdrv_system *s, int idx)
{
    if (!s) return fail(TRPDRV_ERR_ARG, "system %d: NULL descriptor", idx);
    if (s->nocc < 1 || s->nocc > TRPDRV_MAX_NOCC)
        return fail(TRPDRV_ERR_ARG, "system %d: nocc=%d outside [1,%d]", idx, s->nocc, TRPDRV_MAX_NOCC);
    if (s->nvir < 1 || s->nvir > TRPDRV_MAX_NVIR)
        return fail(TRPDRV_ERR_ARG, "system %d: nvir=%d outside [1,%d]", idx, s->nvir, TRPDRV_MAX_NVIR);
    if (s->ncor < 0) return fail(TRPDRV_ERR_ARG, "system %d: ncor=%d < 0", idx, s->ncor);
    const int nbf = s->ncor + s->nocc + s->nvir;
    if (s->a < 1 || s->a > nbf) return fail(TRPDRV_ERR_ARG, "system %d: a=%d outside [1,%d]", idx, s->a, nbf);
    return TRPDRV_OK;
}

static const double *sys_tensor(const trpdrv_system *s, int w)
{
    switch (w) {
    case TRPDRV_T_EORB: return s->eorb;
    case TRPDRV_T_T2: return s->t2;
    case TRPDRV_T_JVV: return s->jvv;
    case TRPDRV_T_KVV: return s->kvv;
    case TRPDRV_T_TOV: return s->tov;
    case TRPDRV_T_XOV: return s->xov;
    case TRPDRV_T_JOV: return s->jov;
    case TRPDRV_T_KOV: return s->kov;
    case TRPDRV_T_DINTC: return s->dintc;
    case TRPDRV_T_DINTX: return s->dintx;
    case TRPDRV_T_T1V: return s->t1v;
    default: return NULL;
    }
}

static int pack_triple(int i, int j, int k) { return (i - 1) | ((j - 1) << 10) | ((k - 1) << 20); }

/* ------------------------------------------------------------------------------------------ */
/* plans                                                                                        */
/* ------------------------------------------------------------------------------------------ */

#define TUNE_MAX_BATCH 64 /* largest emulated batch the autotuner tries */

typedef struct sysbuf {
    trpdrv_system shape;
    const double *t[TRPDRV_T_COUNT]; /* device tensors in use (owned or bound) */
    double *own[TRPDRV_T_COUNT];     /* owned device copies made by upload */
    double *ntov, *nxov;             /* -tov, -xov (rows of ldv doubles when padded) */
    double *pad[TRPDRV_T_COUNT];     /* fused, cp.async staging: t2, jvv, kvv, jov, kov with rows padded to an even
                                        length, refilled by every execution from the bound tensors */
    int32_t *d_triples, *h_triples;
    int32_t *d_order;                /* fused/emulated processing order (trpdrv_processing_order) */
    int32_t *h_order;                /* its host copy (chunks of trpdrv_plan_upload_execute) */
    trpdrv_oz_system oz;             /* emulated form: digit slices and scales (device) */
    int64_t *oz_job0;                /* emulated form: first entry of oz.jobs of each position */
    void *oz_maps;                   /* emulated form: tensor maps of oz.sa / oz.sb (host blob) */
    int64_t ntriples;                /* records: n_a * nt */
    int64_t nt;                      /* triples per a (this rank's share) */
    int n_a;                         /* virtual indices swept (options.a_count) */
    double *partial, *rec;
    int nb, npairs;
} sysbuf;

struct trpdrv_plan {
    int nsys, device, nsm, grid, grid_tma, vec2, bound;
    int padded;         /* FUSED: the cp.async staging reads row-padded copies (sysbuf.pad) */
    trpdrv_options opt;
    cudaStream_t stream;
    sysbuf *s;
    trpdrv_dev_system *h_dev, *d_dev;
    unsigned long long *d_counter; /* work tickets and, 8 bytes on, the status word: cleared together */
    int *d_status;
    double *d_bsum;   /* block sums of the totals */
    unsigned *d_done; /* finished blocks per system */
    double *h_res;    /* pinned (res_take): totals per system (emp4 hi, lo, emp5 hi, lo), then the status word */
    double *d_res;    /* its device address */
    int res_own;      /* h_res is pages of this plan's own */
    int64_t total_items;
    double *d_f, *d_bpart; /* plain form: f and energy partials of one batch of triples */
    unsigned *d_tcount;
    int plain_cap;         /* the most triples they hold */
    cudaGraph_t graph;
    cudaGraphExec_t gexec;
    int graph_ready;
    cudaEvent_t ev0, ev1;
    int events_valid;
    int64_t last_launches;
    cudaStream_t last_stream;
    int use_tma;        /* the fused launch stages panels with TMA (fused_tma.cu) */
    int tma_mma_k;      /* FP64 MMA shape of the TMA kernel: 8 (m16n8k8) or 16 (m16n8k16) */
    double *d_fbuf;     /* emulated form: f of two batches of triples [2][fbuf_batch][8][nvir][nvir] */
    size_t fbuf_half;   /* doubles in one of the two halves */
    cudaStream_t aux_stream;          /* emulated form: energies of batch n, ordered after its products only */
    cudaEvent_t ev_gemm[2], ev_tengy[2];
    int tengy_sent[2];  /* ev_tengy was recorded by the job being enqueued: what an earlier one recorded, or a
                           capture, is not waited for */
    int fbuf_batch;     /* triples d_fbuf holds (>= opt.batch, and room for the autotuner's batches) */
    int tuned_staging;  /* FUSED staging chosen by the autotuner (1 cp.async, 2 TMA), 0 = none */
    void *tma_maps;     /* tensor maps of every system, passed by value to each launch */
    /* trpdrv_plan_upload_execute: copy stream, one event per chunk, the chunks' first work items */
    cudaStream_t copy_stream;
    cudaEvent_t *chunk_ev, ev_in, ev_out;
    int nchunk_ev;
    unsigned long long *d_chunk_first, *h_chunk_first;
    int nchunk_first;
};

void trpdrv_options_default(trpdrv_options *opt)
{
    if (!opt) return;
    memset(opt, 0, sizeof *opt);
    opt->mode = TRPDRV_MODE_FUSED;
    opt->nkpass = 1;
    opt->rank = 0;
    opt->world = 1;
    opt->device = -1;
    opt->tile = 0;
    opt->ctas_per_sm = 0;
    opt->use_graph = 1;
    opt->mma_k = 8;
    opt->slices = 7;
    opt->batch = 64;
}

/* ------------------------------------------------------------------------------------------ */
/* pinned memory for the plans' totals                                                          */
/* ------------------------------------------------------------------------------------------ */

/* One pinned block for the whole process, of which every plan takes a few 64-byte lines for as long as it lives:
 * pinning memory of its own (0.25 ms, and as much to give it back) doubled the creation of a small plan, which a caller
 * of trpdrv_run pays on every call.  trpdrv_finalize frees it, or the last plan does that is left then.  Plans of
 * more systems than there is room for pin pages of their own. */
enum { RES_LINE = 8, RES_LINES = 512 }; /* doubles per line; 32 KB */
static pthread_mutex_t g_res_mu = PTHREAD_MUTEX_INITIALIZER;
static double *g_res;
static unsigned char g_res_taken[RES_LINES];
static int g_res_plans, g_res_closing;

/* Room for n doubles, zeroed; *own: pages of this plan alone. */
static int res_take(size_t n, double **out, int *own)
{
    const size_t lines = (n + RES_LINE - 1) / RES_LINE;
    *out = NULL;
    *own = 0;
    pthread_mutex_lock(&g_res_mu);
    cudaError_t e = cudaSuccess;
    if (lines <= RES_LINES && !g_res)
        e = cudaHostAlloc((void **)&g_res, sizeof(double) * RES_LINE * RES_LINES,
                          cudaHostAllocPortable | cudaHostAllocMapped);
    if (e == cudaSuccess && lines <= RES_LINES) {
        size_t run = 0;
        for (size_t l = 0; l < RES_LINES && run < lines; ++l) {
            run = g_res_taken[l] ? 0 : run + 1;
            if (run == lines) {
                *out = g_res + RES_LINE * (l + 1 - lines);
                memset(g_res_taken + (l + 1 - lines), 1, lines);
                ++g_res_plans;
                g_res_closing = 0;
            }
        }
    }
    pthread_mutex_unlock(&g_res_mu);
    CUDA_TRY(e);
    if (!*out) {
        const size_t bytes = (sizeof(double) * n + 4095) / 4096 * 4096;
        void *pages = aligned_alloc(4096, bytes);
        if (!pages) return fail(TRPDRV_ERR_NOMEM, "out of host memory");
        e = cudaHostRegister(pages, bytes, cudaHostRegisterPortable | cudaHostRegisterMapped);
        if (e != cudaSuccess) free(pages);
        CUDA_TRY(e);
        *out = (double *)pages;
        *own = 1;
    }
    memset(*out, 0, sizeof(double) * n);
    return TRPDRV_OK;
}

/* with g_res_mu held */
static void res_free_unused(void)
{
    if (g_res && g_res_plans == 0) {
        cudaFreeHost(g_res);
        g_res = NULL;
    }
}

/* No kernel writes there any more. */
static void res_give(double *res, size_t n, int own)
{
    if (!res) return;
    if (own) {
        cudaHostUnregister(res);
        free(res);
        return;
    }
    pthread_mutex_lock(&g_res_mu);
    memset(g_res_taken + (res - g_res) / RES_LINE, 0, (n + RES_LINE - 1) / RES_LINE);
    --g_res_plans;
    if (g_res_closing) res_free_unused();
    pthread_mutex_unlock(&g_res_mu);
}

static void res_close(void)
{
    pthread_mutex_lock(&g_res_mu);
    g_res_closing = 1;
    res_free_unused();
    pthread_mutex_unlock(&g_res_mu);
}

static size_t res_doubles(const trpdrv_plan *p) { return 4 * (size_t)p->nsys + 1; }

static void plan_free(trpdrv_plan *p)
{
    if (!p) return;
    if (p->gexec) cudaGraphExecDestroy(p->gexec);
    if (p->graph) cudaGraphDestroy(p->graph);
    if (p->s) {
        for (int q = 0; q < p->nsys; ++q) {
            sysbuf *b = &p->s[q];
            for (int w = 0; w < TRPDRV_T_COUNT; ++w)
                if (b->own[w]) cudaFree(b->own[w]);
            for (int w = 0; w < TRPDRV_T_COUNT; ++w)
                if (b->pad[w]) cudaFree(b->pad[w]);
            if (b->ntov) cudaFree(b->ntov);
            if (b->nxov) cudaFree(b->nxov);
            if (b->d_triples) cudaFree(b->d_triples);
            if (b->d_order) cudaFree(b->d_order);
            free(b->h_order);
            if (b->oz.sa) cudaFree(b->oz.sa);
            if (b->oz.sb) cudaFree(b->oz.sb);
            if (b->oz.ea) cudaFree(b->oz.ea);
            if (b->oz.eb) cudaFree(b->oz.eb);
            if (b->oz.jobs) cudaFree(b->oz.jobs);
            free(b->oz_job0);
            free(b->oz_maps);
            if (b->partial) cudaFree(b->partial);
            if (b->rec) cudaFree(b->rec);
            free(b->h_triples);
        }
        free(p->s);
    }
    free(p->h_dev);
    free(p->tma_maps);
    if (p->d_dev) cudaFree(p->d_dev);
    if (p->d_counter) cudaFree(p->d_counter);
    if (p->d_bsum) cudaFree(p->d_bsum);
    if (p->d_done) cudaFree(p->d_done);
    if (p->d_f) cudaFree(p->d_f);
    if (p->d_fbuf) cudaFree(p->d_fbuf);
    for (int h = 0; h < 2; ++h) {
        if (p->ev_gemm[h]) cudaEventDestroy(p->ev_gemm[h]);
        if (p->ev_tengy[h]) cudaEventDestroy(p->ev_tengy[h]);
    }
    if (p->aux_stream) cudaStreamDestroy(p->aux_stream);
    if (p->d_bpart) cudaFree(p->d_bpart);
    if (p->d_tcount) cudaFree(p->d_tcount);
    if (p->ev0) cudaEventDestroy(p->ev0);
    if (p->ev1) cudaEventDestroy(p->ev1);
    for (int c = 0; c < p->nchunk_ev; ++c) cudaEventDestroy(p->chunk_ev[c]);
    free(p->chunk_ev);
    if (p->ev_in) cudaEventDestroy(p->ev_in);
    if (p->ev_out) cudaEventDestroy(p->ev_out);
    if (p->d_chunk_first) cudaFree(p->d_chunk_first);
    free(p->h_chunk_first);
    if (p->copy_stream) cudaStreamDestroy(p->copy_stream);
    if (p->stream) cudaStreamDestroy(p->stream);
    if (p->last_stream) cudaDeviceSynchronize(); /* an execution nobody waited for still writes its totals */
    res_give(p->h_res, res_doubles(p), p->res_own);
    free(p);
}

/* Triples per launch of a plain plan's system: at most `cap`. */
static int64_t plain_batch(const sysbuf *b, int cap)
{
    int64_t n = trpdrv_plain_batch(b->shape.nvir);
    if (n > cap) n = cap;
    return b->ntriples < n ? (b->ntriples > 0 ? b->ntriples : 1) : n;
}

/* The buffers of one batch of the largest system, f and energy partials.  f of a full batch is 96 MB.  The plan's own
 * tensors and whatever the application holds come after it, so f takes a quarter of the free memory at most (asked for
 * above 4 MB: the question takes 0.1 ms): batches are halved until it does and the allocation succeeds, down to the
 * single triple that a plan cannot do without. */
static int plain_buffers(trpdrv_plan *p)
{
    size_t limit = (size_t)4 << 20;
    int asked = 0;
    for (p->plain_cap = 256;; p->plain_cap /= 2) {
        size_t nf = 1, nbp = 1, nct = 1;
        for (int q = 0; q < p->nsys; ++q) {
            const size_t V = (size_t)p->s[q].shape.nvir, n = (size_t)plain_batch(&p->s[q], p->plain_cap);
            if (n * 8 * V * V > nf) nf = n * 8 * V * V;
            if (n * 4 * (size_t)trpdrv_tengy_pairs((int)V) > nbp) nbp = n * 4 * (size_t)trpdrv_tengy_pairs((int)V);
            if (n > nct) nct = n;
        }
        if (sizeof(double) * nf > limit && !asked) {
            size_t avail = 0, total = 0;
            CUDA_TRY(cudaMemGetInfo(&avail, &total));
            if (avail / 4 > limit) limit = avail / 4;
            asked = 1;
        }
        if (sizeof(double) * nf > limit && p->plain_cap > 1) continue;
        cudaError_t e = cudaMalloc((void **)&p->d_f, sizeof(double) * nf);
        if (e == cudaSuccess) e = cudaMalloc((void **)&p->d_bpart, sizeof(double) * nbp);
        if (e == cudaSuccess) e = cudaMalloc((void **)&p->d_tcount, sizeof(unsigned) * nct);
        if (e == cudaSuccess) e = cudaMemset(p->d_tcount, 0, sizeof(unsigned) * nct);
        if (e == cudaSuccess) return TRPDRV_OK;
        if (e != cudaErrorMemoryAllocation || p->plain_cap == 1) CUDA_TRY(e);
        cudaGetLastError();
        if (p->d_f) cudaFree(p->d_f);
        if (p->d_bpart) cudaFree(p->d_bpart);
        if (p->d_tcount) cudaFree(p->d_tcount);
        p->d_f = p->d_bpart = NULL;
        p->d_tcount = NULL;
    }
}

static int plan_build(trpdrv_plan *p, const trpdrv_system *shape)
{
    const trpdrv_options *o = &p->opt;
    CUDA_TRY(cudaStreamCreateWithFlags(&p->stream, cudaStreamNonBlocking));
    CUDA_TRY(cudaEventCreate(&p->ev0));
    CUDA_TRY(cudaEventCreate(&p->ev1));
    p->s = (sysbuf *)calloc((size_t)p->nsys, sizeof(sysbuf));
    p->h_dev = (trpdrv_dev_system *)calloc((size_t)p->nsys, sizeof(trpdrv_dev_system));
    if (!p->s || !p->h_dev) return fail(TRPDRV_ERR_NOMEM, "host allocation failed");

    int64_t item = 0;
    int maxv = 0;
    int even = 1;
    for (int q = 0; q < p->nsys; ++q) {
        sysbuf *b = &p->s[q];
        b->shape = shape[q];
        const int nocc = shape[q].nocc, nvir = shape[q].nvir;
        if ((nocc & 1) || (nvir & 1)) even = 0;
        b->nb = (nvir + TRPDRV_TILE - 1) / TRPDRV_TILE;
        b->npairs = b->nb * (b->nb + 1) / 2;
        if (nvir > maxv) maxv = nvir;

        /* the reference driver's order, then this rank's contiguous share (uniform cost per system) */
        const int64_t n = trpdrv_shard_triples(nocc, o->nkpass, o->rank, o->world, NULL);
        if (n < 0) return fail(TRPDRV_ERR_ARG, "system %d: cannot shard triples", q);
        b->nt = n;
        b->n_a = o->a_count;
        b->ntriples = n * o->a_count;
        if (b->ntriples > INT32_MAX) return fail(TRPDRV_ERR_ARG, "system %d: more than 2^31 (a, triple) records", q);
        int32_t *ijk = (int32_t *)malloc(sizeof(int32_t) * 3 * (size_t)(n > 0 ? n : 1));
        b->h_triples = (int32_t *)malloc(sizeof(int32_t) * (size_t)(n > 0 ? n : 1));
        if (!ijk || !b->h_triples) {
            free(ijk);
            return fail(TRPDRV_ERR_NOMEM, "host allocation failed");
        }
        trpdrv_shard_triples(nocc, o->nkpass, o->rank, o->world, ijk);
        for (int64_t t = 0; t < n; ++t) b->h_triples[t] = pack_triple(ijk[3 * t], ijk[3 * t + 1], ijk[3 * t + 2]);
        int32_t *order = NULL;
        if (o->mode != TRPDRV_MODE_PLAIN && n > 0) {
            order = (int32_t *)malloc(sizeof(int32_t) * (size_t)n);
            if (!order || trpdrv_processing_order(ijk, n, 0, order) != 0) {
                free(order);
                free(ijk);
                return fail(TRPDRV_ERR_NOMEM, "host allocation failed");
            }
        }
        free(ijk);
        if (order) {
            const cudaError_t e1 = cudaMalloc((void **)&b->d_order, sizeof(int32_t) * (size_t)n);
            const cudaError_t e2 = e1 == cudaSuccess ? cudaMemcpy(b->d_order, order, sizeof(int32_t) * (size_t)n,
                                                                  cudaMemcpyHostToDevice)
                                                     : e1;
            b->h_order = order;
            CUDA_TRY(e2);
        }

        if (b->ntriples > 0) {
            CUDA_TRY(cudaMalloc((void **)&b->d_triples, sizeof(int32_t) * (size_t)b->nt));
            CUDA_TRY(cudaMemcpy(b->d_triples, b->h_triples, sizeof(int32_t) * (size_t)b->nt,
                                cudaMemcpyHostToDevice));
            CUDA_TRY(cudaMalloc((void **)&b->rec, sizeof(double) * 4 * (size_t)b->ntriples));
            CUDA_TRY(cudaMemset(b->rec, 0, sizeof(double) * 4 * (size_t)b->ntriples));
            if (o->mode != TRPDRV_MODE_PLAIN) {
                const size_t pb = sizeof(double) * 4 * TRPDRV_FUSED_SLOTS * (size_t)b->ntriples * b->npairs;
                CUDA_TRY(cudaMalloc((void **)&b->partial, pb));
                /* the emulated form writes only some slots of each item; the rest stay zero */
                CUDA_TRY(cudaMemset(b->partial, 0, pb));
            }
        }
        if (o->mode == TRPDRV_MODE_EMULATED) {
            trpdrv_oz_system *z = &b->oz;
            z->nocc = nocc;
            z->nvir = nvir;
            z->slices = o->slices;
            z->dp = trpdrv_oz_dp(nocc, nvir);
            z->n_a = o->a_count;
            const size_t rows = 2 * (size_t)nvir, per = (size_t)o->slices * rows * (size_t)z->dp;
            CUDA_TRY(cudaMalloc((void **)&z->sa, per * (size_t)nocc * (size_t)z->n_a));
            CUDA_TRY(cudaMalloc((void **)&z->sb, per * (size_t)nocc * nocc));
            CUDA_TRY(cudaMalloc((void **)&z->ea, sizeof(double) * rows * (size_t)nocc * (size_t)z->n_a));
            CUDA_TRY(cudaMalloc((void **)&z->eb, sizeof(double) * rows * (size_t)nocc * nocc));
            /* the products of every record position; a position's first job: oz_job0 */
            const int64_t nr = b->ntriples;
            int32_t *jobs = (int32_t *)malloc(sizeof(int32_t) * (size_t)(2 * nr + 1));
            b->oz_job0 = (int64_t *)malloc(sizeof(int64_t) * (size_t)(nr + 1));
            if (!jobs || !b->oz_job0 || nr > INT32_MAX / 2) {
                free(jobs);
                return nr > INT32_MAX / 2 ? fail(TRPDRV_ERR_ARG, "system %d: more than 2^30 (a, triple) records", q)
                                          : fail(TRPDRV_ERR_NOMEM, "host allocation failed");
            }
            int64_t nj = 0;
            for (int64_t r = 0; r < nr; ++r) {
                const int64_t t = r % b->nt;
                const int pk = b->h_triples[b->h_order ? b->h_order[t] : t];
                b->oz_job0[r] = nj;
                jobs[nj++] = (int32_t)(r << 1);
                if ((pk & 1023) != ((pk >> 20) & 1023)) jobs[nj++] = (int32_t)(r << 1 | 1);
            }
            b->oz_job0[nr] = nj;
            cudaError_t je = cudaMalloc((void **)&z->jobs, sizeof(int32_t) * (size_t)(nj + 1));
            if (je == cudaSuccess)
                je = cudaMemcpy(z->jobs, jobs, sizeof(int32_t) * (size_t)nj, cudaMemcpyHostToDevice);
            free(jobs);
            CUDA_TRY(je);
            b->oz_maps = aligned_alloc(64, (trpdrv_oz_maps_bytes() + 63) & ~(size_t)63);
            if (!b->oz_maps) return fail(TRPDRV_ERR_NOMEM, "host allocation failed");
        }
        const size_t ovp = (size_t)nocc * nocc * (size_t)(nvir + (nvir & 1)); /* room for padded rows */
        CUDA_TRY(cudaMalloc((void **)&b->ntov, sizeof(double) * ovp));
        CUDA_TRY(cudaMalloc((void **)&b->nxov, sizeof(double) * ovp));

        trpdrv_dev_system *d = &p->h_dev[q];
        d->ncor = shape[q].ncor;
        d->nocc = nocc;
        d->nvir = nvir;
        d->a = shape[q].a;
        d->nb = b->nb;
        d->npairs = b->npairs;
        d->pack_edge = trpdrv_tma_pack_edge(nvir);
        d->ntriples = b->ntriples;
        d->nt = b->nt;
        d->n_a = b->n_a;
        d->item_begin = item;
        d->triples = b->d_triples;
        d->order = b->d_order;
        d->partial = b->partial;
        d->rec = b->rec;
        d->ntov = b->ntov;
        d->nxov = b->nxov;
        item += b->ntriples * b->npairs;
    }
    p->total_items = item;
    p->vec2 = even;
    CUDA_TRY(cudaMalloc((void **)&p->d_dev, sizeof(trpdrv_dev_system) * (size_t)p->nsys));
    CUDA_TRY(cudaMalloc((void **)&p->d_counter, 2 * sizeof(unsigned long long)));
    CUDA_TRY(cudaMemset(p->d_counter, 0, 2 * sizeof(unsigned long long)));
    p->d_status = (int *)(p->d_counter + 1);
    CUDA_TRY(cudaMalloc((void **)&p->d_bsum, sizeof(double) * (trpdrv_totals_doubles(p->h_dev, p->nsys) + 1)));
    CUDA_TRY(cudaMalloc((void **)&p->d_done, sizeof(unsigned) * (size_t)p->nsys));
    CUDA_TRY(cudaMemset(p->d_done, 0, sizeof(unsigned) * (size_t)p->nsys));
    TRY(res_take(res_doubles(p), &p->h_res, &p->res_own));
    CUDA_TRY(cudaHostGetDevicePointer((void **)&p->d_res, p->h_res, 0));
    if (o->mode == TRPDRV_MODE_EMULATED) {
        p->fbuf_batch = o->batch > TUNE_MAX_BATCH ? o->batch : TUNE_MAX_BATCH;
        p->fbuf_half = 8 * (size_t)p->fbuf_batch * maxv * trpdrv_oz_ldf(maxv);
        CUDA_TRY(cudaMalloc((void **)&p->d_fbuf, sizeof(double) * 2 * p->fbuf_half));
        CUDA_TRY(cudaStreamCreateWithFlags(&p->aux_stream, cudaStreamNonBlocking));
        for (int h = 0; h < 2; ++h) {
            CUDA_TRY(cudaEventCreateWithFlags(&p->ev_gemm[h], cudaEventDisableTiming));
            CUDA_TRY(cudaEventCreateWithFlags(&p->ev_tengy[h], cudaEventDisableTiming));
        }
    }
    if (o->mode == TRPDRV_MODE_PLAIN) TRY(plain_buffers(p));

    int per_sm = o->ctas_per_sm;
    if (per_sm <= 0) per_sm = 1; /* the fused kernel's stages fill an SM's shared memory */
    int64_t grid = (int64_t)per_sm * p->nsm;
    if (grid > p->total_items) grid = p->total_items;
    p->grid = (int)(grid > 0 ? grid : 0);
    int64_t grid_tma = p->nsm; /* fused_tma.cu: one CTA per SM */
    if (grid_tma > p->total_items) grid_tma = p->total_items;
    p->grid_tma = (int)(grid_tma > 0 ? grid_tma : 0);
    return TRPDRV_OK;
}

int trpdrv_plan_create(trpdrv_plan **plan, const trpdrv_system *shape, int nsys, const trpdrv_options *opt)
{
    if (!plan) return fail(TRPDRV_ERR_ARG, "plan output pointer is NULL");
    *plan = NULL;
    if (nsys < 1 || !shape) return fail(TRPDRV_ERR_ARG, "nsys=%d / shape=%p", nsys, (const void *)shape);
    trpdrv_options o;
    if (opt)
        o = *opt;
    else
        trpdrv_options_default(&o);
    if (o.mode != TRPDRV_MODE_PLAIN && o.mode != TRPDRV_MODE_FUSED && o.mode != TRPDRV_MODE_EMULATED)
        return fail(TRPDRV_ERR_ARG, "unknown mode %d", o.mode);
    if (o.target_digits < 0 || o.target_digits > 15)
        return fail(TRPDRV_ERR_ARG, "target_digits %d: must be 0..15", o.target_digits);
    if (o.slices == 0) o.slices = 7;
    if (o.mode == TRPDRV_MODE_EMULATED && o.target_digits > 0) o.slices = 8; /* room for any choice */
    if (o.batch == 0) o.batch = 64;
    if (!trpdrv_oz_slices_supported(o.slices))
        return fail(TRPDRV_ERR_ARG, "slices %d: must be %d..%d", o.slices, TRPDRV_OZ_MIN_SLICES, TRPDRV_OZ_MAX_SLICES);
    if (o.batch < 1 || o.batch > 4096) return fail(TRPDRV_ERR_ARG, "batch %d: must be 1..4096", o.batch);
    if (o.a_count == 0) o.a_count = 1;
    if (o.a_count < 1 || o.a_count > 1023) return fail(TRPDRV_ERR_ARG, "a_count %d: must be 1..1023", o.a_count);
    if (o.world < 1 || o.rank < 0 || o.rank >= o.world)
        return fail(TRPDRV_ERR_ARG, "rank %d / world %d", o.rank, o.world);
    if (o.tile != 0 && o.tile != TRPDRV_TILE)
        return fail(TRPDRV_ERR_UNSUPPORTED, "tile %d: only %d is compiled", o.tile, TRPDRV_TILE);
    if (o.nkpass < 1) o.nkpass = 1;
    if (o.mma_k == 0) o.mma_k = 8;
    if (o.mma_k != 4 && o.mma_k != 8 && o.mma_k != 16)
        return fail(TRPDRV_ERR_ARG, "mma_k %d: must be 4, 8 or 16", o.mma_k);
    if (o.staging < 0 || o.staging > 2) return fail(TRPDRV_ERR_ARG, "staging %d: must be 0, 1 or 2", o.staging);
    for (int q = 0; q < nsys; ++q) {
        TRY(check_shape(&shape[q], q));
        const int nbf = shape[q].ncor + shape[q].nocc + shape[q].nvir;
        if (shape[q].a + o.a_count - 1 > nbf)
            return fail(TRPDRV_ERR_ARG, "system %d: a=%d with a_count=%d passes the basis size %d", q, shape[q].a,
                        o.a_count, nbf);
    }

    int dev = 0, nsm = 0;
    TRY(ensure_device(o.device, &dev, &nsm));
    trpdrv_plan *p = (trpdrv_plan *)calloc(1, sizeof(trpdrv_plan));
    if (!p) return fail(TRPDRV_ERR_NOMEM, "host allocation failed");
    p->nsys = nsys;
    p->opt = o;
    /* mma_k names the shape of whichever fused kernel runs: 16 exists only with TMA staging, 4 only
     * with cp.async staging; each kernel takes its nearest shape */
    p->tma_mma_k = o.mma_k == 16 ? 16 : 8;
    if (p->opt.mma_k == 16) p->opt.mma_k = 8;
    p->device = dev;
    p->nsm = nsm;
    int rc = plan_build(p, shape);
    if (rc != TRPDRV_OK) {
        const int st = t_status;
        char msg[sizeof t_message];
        memcpy(msg, t_message, sizeof msg);
        plan_free(p);
        t_status = st;
        memcpy(t_message, msg, sizeof msg);
        return rc;
    }
    *plan = p;
    return TRPDRV_OK;
}

/* Doubles per row and rows of tensor w of system b as the kernels read it (t2, jvv, kvv: rows of nvir; jov,
 * kov: rows of nocc). */
static int tensor_rows(const sysbuf *b, int w, long long *rows)
{
    const long long O = b->shape.nocc, V = b->shape.nvir;
    switch (w) {
    case TRPDRV_T_T2: *rows = O * O * V; return (int)V;
    case TRPDRV_T_JVV:
    case TRPDRV_T_KVV: *rows = b->n_a * O * V; return (int)V;
    case TRPDRV_T_JOV:
    case TRPDRV_T_KOV: *rows = O * O * V; return (int)O;
    default: *rows = 0; return 0;
    }
}

static int row_pitch(int width) { return width + (width & 1); }

/* Bytes of the padded copy that tensor w of system b needs for 16-byte copies and does not have yet. */
static size_t pad_bytes(const sysbuf *b, int w)
{
    long long rows;
    const int width = tensor_rows(b, w, &rows);
    if (!width || rows == 0 || b->pad[w]) return 0;
    if (!(width & 1) && !(((uintptr_t)b->t[w]) & 15u)) return 0;
    return sizeof(double) * (size_t)rows * row_pitch(width);
}

/* Fused plans that cannot copy 16 bytes at a time from the bound tensors (an odd nvir or nocc, or an
 * unaligned pointer) and do not use TMA: the tensors concerned get copies with rows padded to an even length
 * (zero pads), which every execution refills.  Copying each input once costs little beside the kernel, which
 * reads a block of T2 for every triple: (13, 151) runs 4.2 ms with 8-byte copies from the bound tensors.
 * The copies take as much memory as those tensors.  The caller did not ask for them, so they are made only out of
 * plenty: a quarter of the memory that is free at this moment, at most (asked for above 16 MB: the question takes
 * 0.1 ms, as long as a small plan's execution).  Else, or where the allocation fails, the kernel reads the bound
 * tensors with 8-byte copies. */
#define PAD_FREELY ((size_t)16 << 20)
static int plan_pad(trpdrv_plan *p, int tma_ok)
{
    p->padded = 0;
    for (int q = 0; q < p->nsys; ++q) p->h_dev[q].ldv = p->h_dev[q].ldo = 0;
    if (p->opt.mode != TRPDRV_MODE_FUSED || p->vec2 || tma_ok) return TRPDRV_OK;
    size_t need = 0;
    for (int q = 0; q < p->nsys; ++q)
        for (int w = 0; w < TRPDRV_T_COUNT; ++w) need += pad_bytes(&p->s[q], w);
    int ok = 1;
    if (need > PAD_FREELY) {
        size_t avail = 0, total = 0;
        CUDA_TRY(cudaMemGetInfo(&avail, &total));
        ok = need <= avail / 4;
    }
    for (int q = 0; q < p->nsys && ok; ++q) {
        sysbuf *b = &p->s[q];
        for (int w = 0; w < TRPDRV_T_COUNT && ok; ++w) {
            const size_t bytes = pad_bytes(b, w);
            if (bytes == 0) continue;
            if (cudaMalloc((void **)&b->pad[w], bytes) != cudaSuccess) {
                b->pad[w] = NULL;
                cudaGetLastError();
                ok = 0;
            }
        }
    }
    if (!ok) {
        for (int q = 0; q < p->nsys; ++q)
            for (int w = 0; w < TRPDRV_T_COUNT; ++w) {
                if (p->s[q].pad[w]) cudaFree(p->s[q].pad[w]);
                p->s[q].pad[w] = NULL;
            }
        return TRPDRV_OK;
    }
    p->padded = 1;
    return TRPDRV_OK;
}

/* Whether tensor w of system q is read through its padded copy. */
static int reads_pad(const trpdrv_plan *p, int q, int w)
{
    long long rows;
    const sysbuf *b = &p->s[q];
    const int width = tensor_rows(b, w, &rows);
    return p->padded && width && b->pad[w] && ((width & 1) || (((uintptr_t)b->t[w]) & 15u));
}

static const double *fused_tensor(const trpdrv_plan *p, int q, int w)
{
    return reads_pad(p, q, w) ? p->s[q].pad[w] : p->s[q].t[w];
}

/* Refills padded copies of system q from its tensors: those every j reads (want_all), and blocks
 * jlo <= j < jhi of the others. */
static int pad_refill(trpdrv_plan *p, int q, int want_all, int jlo, int jhi, cudaStream_t st, int64_t *launches)
{
    if (!p->padded || p->use_tma) return TRPDRV_OK;
    const sysbuf *b = &p->s[q];
    trpdrv_pack_list L;
    memset(&L, 0, sizeof L);
    for (int w = 0; w < TRPDRV_T_COUNT; ++w) {
        if (!reads_pad(p, q, w)) continue;
        const int byj = w == TRPDRV_T_T2 || w == TRPDRV_T_JOV || w == TRPDRV_T_KOV;
        if (byj ? jlo >= jhi : !want_all) continue;
        long long rows, first = 0;
        const int width = tensor_rows(b, w, &rows);
        if (byj) {
            const long long per_j = (long long)b->shape.nocc * b->shape.nvir;
            first = jlo * per_j;
            rows = (jhi - jlo) * per_j;
        }
        L.seg[L.n].src = b->t[w] + first * width;
        L.seg[L.n].dst = b->pad[w] + first * row_pitch(width);
        L.seg[L.n].rows = rows;
        L.seg[L.n].width = width;
        L.seg[L.n].pitch = row_pitch(width);
        ++L.n;
    }
    if (!L.n) return TRPDRV_OK;
    LAUNCH_TRY(trpdrv_launch_pack_rows(&L, st));
    if (launches) ++*launches;
    return TRPDRV_OK;
}

static int plan_publish(trpdrv_plan *p)
{
    /* TMA reads the bound tensors themselves */
    for (int q = 0; q < p->nsys; ++q) {
        p->h_dev[q].t2 = p->s[q].t[TRPDRV_T_T2];
        p->h_dev[q].jvv = p->s[q].t[TRPDRV_T_JVV];
        p->h_dev[q].kvv = p->s[q].t[TRPDRV_T_KVV];
        p->h_dev[q].jov = p->s[q].t[TRPDRV_T_JOV];
        p->h_dev[q].kov = p->s[q].t[TRPDRV_T_KOV];
    }
    const int want = p->opt.staging;
    const int tma_ok = p->opt.mode == TRPDRV_MODE_FUSED && want != 1 && trpdrv_tma_supported(p->h_dev, p->nsys);
    if (p->opt.mode == TRPDRV_MODE_FUSED && want == 2 && !tma_ok)
        return fail(TRPDRV_ERR_UNSUPPORTED, "TMA staging needs even nvir and nocc, 16-byte aligned tensors "
                                            "and at most %d systems", TRPDRV_TMA_MAX_SYSTEMS);
    TRY(plan_pad(p, tma_ok));
    for (int q = 0; q < p->nsys; ++q) {
        sysbuf *b = &p->s[q];
        trpdrv_dev_system *d = &p->h_dev[q];
        d->eorb = b->t[TRPDRV_T_EORB];
        d->t2 = fused_tensor(p, q, TRPDRV_T_T2);
        d->jvv = fused_tensor(p, q, TRPDRV_T_JVV);
        d->kvv = fused_tensor(p, q, TRPDRV_T_KVV);
        d->jov = fused_tensor(p, q, TRPDRV_T_JOV);
        d->kov = fused_tensor(p, q, TRPDRV_T_KOV);
        d->dintc = b->t[TRPDRV_T_DINTC];
        d->dintx = b->t[TRPDRV_T_DINTX];
        d->t1v = b->t[TRPDRV_T_T1V];
        const int O = b->shape.nocc, V = b->shape.nvir;
        if (p->padded) { /* one pitch per dimension: even sizes keep theirs */
            d->ldv = row_pitch(V);
            d->ldo = row_pitch(O);
        }
        trpdrv_pack_list N;
        memset(&N, 0, sizeof N);
        if (p->padded) {
            N.n = 2;
            for (int x = 0; x < 2; ++x) {
                N.seg[x].src = b->t[x ? TRPDRV_T_XOV : TRPDRV_T_TOV];
                N.seg[x].dst = x ? b->nxov : b->ntov;
                N.seg[x].rows = (long long)O * O;
                N.seg[x].width = V;
                N.seg[x].pitch = row_pitch(V);
                N.seg[x].neg = 1;
            }
            LAUNCH_TRY(trpdrv_launch_pack_rows(&N, p->stream));
        } else {
            const size_t ov = (size_t)O * O * V;
            LAUNCH_TRY(trpdrv_launch_negate(b->t[TRPDRV_T_TOV], b->ntov, ov, p->stream));
            LAUNCH_TRY(trpdrv_launch_negate(b->t[TRPDRV_T_XOV], b->nxov, ov, p->stream));
        }
    }
    if (p->opt.mode == TRPDRV_MODE_EMULATED) {
        for (int q = 0; q < p->nsys; ++q) {
            const int e = trpdrv_oz_prepare(&p->s[q].oz, p->s[q].oz_maps);
            if (e) return fail(TRPDRV_ERR_CUDA, "tensor-map encoding failed (%d)", e);
        }
    }
    if (p->opt.mode != TRPDRV_MODE_PLAIN && p->graph_ready) { /* the graph holds the old parameters */
        cudaGraphExecDestroy(p->gexec);
        cudaGraphDestroy(p->graph);
        p->gexec = NULL;
        p->graph = NULL;
        p->graph_ready = 0;
    }
    if (p->opt.mode == TRPDRV_MODE_FUSED) {
        const int ok = tma_ok && p->tuned_staging != 1;
        if (tma_ok) { /* maps whenever TMA is possible, so that the autotuner can time it */
            if (!p->tma_maps) {
                p->tma_maps = aligned_alloc(64, (trpdrv_tma_maps_bytes() + 63) & ~(size_t)63);
                if (!p->tma_maps) return fail(TRPDRV_ERR_NOMEM, "host allocation failed");
            }
            const int e = trpdrv_tma_prepare(p->h_dev, p->nsys, p->tma_maps);
            if (e) return fail(TRPDRV_ERR_CUDA, "tensor-map encoding failed (%d)", e);
        }
        p->use_tma = ok;
    }
    CUDA_TRY(cudaMemcpyAsync(p->d_dev, p->h_dev, sizeof(trpdrv_dev_system) * (size_t)p->nsys,
                             cudaMemcpyHostToDevice, p->stream));
    CUDA_TRY(cudaStreamSynchronize(p->stream));
    p->bound = 1;
    return TRPDRV_OK;
}

/* Elements of tensor w in the plan's device copy (a-dependent tensors hold n_a blocks). */
static size_t upload_elems(const sysbuf *b, int w)
{
    return trpdrv_tensor_elems(w, b->shape.ncor, b->shape.nocc, b->shape.nvir) *
           (trpdrv_tensor_a_dependent(w) ? (size_t)b->n_a : 1);
}

/* Checks `host` against the plan's shapes and allocates the owned device copies it will fill. */
static int upload_prepare(trpdrv_plan *p, const trpdrv_system *host)
{
    for (int q = 0; q < p->nsys; ++q) {
        sysbuf *b = &p->s[q];
        const trpdrv_system *h = &host[q];
        if (h->ncor != b->shape.ncor || h->nocc != b->shape.nocc || h->nvir != b->shape.nvir || h->a != b->shape.a)
            return fail(TRPDRV_ERR_ARG, "system %d: shape differs from the plan's", q);
        for (int w = 0; w < TRPDRV_T_COUNT; ++w) {
            if (!sys_tensor(h, w)) return fail(TRPDRV_ERR_ARG, "system %d: tensor %d is NULL", q, w);
            if (!b->own[w]) CUDA_TRY(cudaMalloc((void **)&b->own[w], sizeof(double) * upload_elems(b, w)));
            b->t[w] = b->own[w];
        }
    }
    return TRPDRV_OK;
}

int trpdrv_plan_upload(trpdrv_plan *p, const trpdrv_system *host, void *stream)
{
    if (!p || !host) return fail(TRPDRV_ERR_ARG, "NULL plan or systems");
    CUDA_TRY(cudaSetDevice(p->device));
    cudaStream_t st = stream ? (cudaStream_t)stream : p->stream;
    TRY(upload_prepare(p, host));
    for (int q = 0; q < p->nsys; ++q)
        for (int w = 0; w < TRPDRV_T_COUNT; ++w)
            CUDA_TRY(cudaMemcpyAsync(p->s[q].own[w], sys_tensor(&host[q], w), sizeof(double) * upload_elems(&p->s[q], w),
                                     cudaMemcpyHostToDevice, st));
    if (st != p->stream) CUDA_TRY(cudaStreamSynchronize(st));
    return plan_publish(p);
}

int trpdrv_plan_bind_device(trpdrv_plan *p, const trpdrv_system *dev)
{
    if (!p || !dev) return fail(TRPDRV_ERR_ARG, "NULL plan or systems");
    CUDA_TRY(cudaSetDevice(p->device));
    int aligned16 = 1;
    for (int q = 0; q < p->nsys; ++q) {
        sysbuf *b = &p->s[q];
        const trpdrv_system *h = &dev[q];
        if (h->ncor != b->shape.ncor || h->nocc != b->shape.nocc || h->nvir != b->shape.nvir || h->a != b->shape.a)
            return fail(TRPDRV_ERR_ARG, "system %d: shape differs from the plan's", q);
        for (int w = 0; w < TRPDRV_T_COUNT; ++w) {
            const double *src = sys_tensor(h, w);
            if (!src) return fail(TRPDRV_ERR_ARG, "system %d: tensor %d is NULL", q, w);
            if (((uintptr_t)src) & 7u) return fail(TRPDRV_ERR_ARG, "system %d: tensor %d not 8-byte aligned", q, w);
            if (((uintptr_t)src) & 15u) aligned16 = 0;
            struct cudaPointerAttributes at;
            if (cudaPointerGetAttributes(&at, src) != cudaSuccess ||
                (at.type != cudaMemoryTypeDevice && at.type != cudaMemoryTypeManaged)) {
                cudaGetLastError();
                return fail(TRPDRV_ERR_ARG, "system %d: tensor %d is not device memory", q, w);
            }
            b->t[w] = src;
        }
    }
    if (!aligned16) p->vec2 = 0;
    return plan_publish(p);
}

/* The records and totals of everything enqueued before on `st`, the totals straight into p->h_res. */
static int enqueue_finish(trpdrv_plan *p, cudaStream_t st, int64_t *launches)
{
    if (p->opt.mode != TRPDRV_MODE_PLAIN) {
        LAUNCH_TRY(trpdrv_launch_records(p->h_dev, p->d_dev, p->nsys, st));
        if (launches) ++*launches;
    }
    LAUNCH_TRY(trpdrv_launch_totals(p->h_dev, p->d_dev, p->nsys, p->d_bsum, p->d_done, p->d_status, p->d_res, st));
    if (launches) ++*launches;
    return TRPDRV_OK;
}

/* Few items per SM: the large ones first.  Inputs this small stay in L2 whatever the order.  (10, 60), 11 items
 * an SM: 133 -> 125 us; (4, 300), 15 an SM: 511 -> 490 us; at 64 and more the two orders time the same. */
static int plan_pair_major(const trpdrv_plan *p) { return p->total_items <= 64 * (int64_t)p->nsm; }

static int enqueue_fused(trpdrv_plan *p, cudaStream_t st, int capturing)
{
    int64_t launches = 0;
    CUDA_TRY(cudaMemsetAsync(p->d_counter, 0, 2 * sizeof(unsigned long long), st)); /* and the status word */
    CUDA_TRY(cudaEventRecordWithFlags(p->ev0, st, capturing ? cudaEventRecordExternal : cudaEventRecordDefault));
    const int pair_major = plan_pair_major(p);
    if (p->total_items > 0) {
        for (int q = 0; q < p->nsys; ++q)
            if (p->h_dev[q].ntriples > 0) TRY(pad_refill(p, q, 1, 0, p->s[q].shape.nocc, st, &launches));
        if (p->use_tma)
            LAUNCH_TRY(trpdrv_launch_fused_tma(p->d_dev, p->nsys, p->total_items, pair_major, p->d_counter,
                                               p->d_status, p->grid_tma, p->tma_maps, p->tma_mma_k, st));
        else
            LAUNCH_TRY(trpdrv_launch_fused(p->d_dev, p->nsys, p->total_items, pair_major, p->d_counter, p->d_status, p->grid,
                                           p->vec2 || p->padded, p->opt.mma_k, st));
        ++launches;
    }
    CUDA_TRY(cudaEventRecordWithFlags(p->ev1, st, capturing ? cudaEventRecordExternal : cudaEventRecordDefault));
    TRY(enqueue_finish(p, st, &launches));
    p->last_launches = launches;
    return TRPDRV_OK;
}

/* Emulated form, positions [pos0, pos1) of one system in batches of `batch`; *bi counts batches over a
 * whole execution (it picks the half of d_fbuf a batch's f goes to).  Even nvir (the default): each
 * contraction launch writes its batch's f into one half while its energy warps compute the energies of
 * the previous batch from the other half, which the previous launch (on the same stream) filled; an
 * energies-only launch closes the system.  Odd nvir, or TRPDRV_OZ_FUSED_ENERGY=0: each batch's
 * energies run as a separate launch on the auxiliary stream while the next batch's
 * products go to the other half; a half is reused only after the energies that read it.  Finish with
 * emulated_join. */
static int emulated_batches(trpdrv_plan *p, const trpdrv_dev_system *d, const sysbuf *b, int64_t pos0, int64_t pos1,
                            int batch, cudaStream_t st, int64_t *bi, int64_t *launches)
{
    if (*bi == 0) p->tengy_sent[0] = p->tengy_sent[1] = 0;
    if (trpdrv_oz_fused_energy_supported(d->nvir)) {
        int64_t epos = 0;
        int en = 0;
        const double *efb = NULL;
        for (int64_t pos = pos0;; pos += batch) {
            const int n = pos < pos1 ? (int)(pos1 - pos < batch ? pos1 - pos : batch) : 0;
            if (n == 0 && en == 0) break;
            const int h = (int)(*bi & 1);
            double *fb = p->d_fbuf + (size_t)h * p->fbuf_half;
            if (n > 0 && p->tengy_sent[h]) CUDA_TRY(cudaStreamWaitEvent(st, p->ev_tengy[h], 0)); /* its separate readers */
            const int64_t j0 = n > 0 ? b->oz_job0[pos] : 0;
            const int nj = n > 0 ? (int)(b->oz_job0[pos + n] - j0) : 0;
            LAUNCH_TRY(trpdrv_launch_oz_gemm(d, &b->oz, b->oz_maps, pos, j0, nj, fb, epos, en, efb, p->d_status,
                                             p->nsm, st));
            if (launches) *launches += 1;
            if (n == 0) break;
            epos = pos;
            en = n;
            efb = fb;
            ++*bi;
        }
        return TRPDRV_OK;
    }
    for (int64_t pos = pos0; pos < pos1; pos += batch) {
        const int n = (int)(pos1 - pos < batch ? pos1 - pos : batch);
        const int h = (int)(*bi & 1);
        double *fb = p->d_fbuf + (size_t)h * p->fbuf_half;
        if (p->tengy_sent[h]) CUDA_TRY(cudaStreamWaitEvent(st, p->ev_tengy[h], 0));
        LAUNCH_TRY(trpdrv_launch_oz_gemm(d, &b->oz, b->oz_maps, pos, b->oz_job0[pos],
                                         (int)(b->oz_job0[pos + n] - b->oz_job0[pos]), fb, 0, 0, NULL, p->d_status,
                                         p->nsm, st));
        CUDA_TRY(cudaEventRecord(p->ev_gemm[h], st));
        CUDA_TRY(cudaStreamWaitEvent(p->aux_stream, p->ev_gemm[h], 0));
        LAUNCH_TRY(trpdrv_launch_oz_tengy(d, pos, n, fb, p->d_status, p->aux_stream));
        CUDA_TRY(cudaEventRecord(p->ev_tengy[h], p->aux_stream));
        p->tengy_sent[h] = 1;
        ++*bi;
        if (launches) *launches += 2;
    }
    return TRPDRV_OK;
}

/* the main stream waits for every energy launch of the batches enqueued so far */
static int emulated_join(trpdrv_plan *p, cudaStream_t st)
{
    for (int h = 0; h < 2; ++h)
        if (p->tengy_sent[h]) CUDA_TRY(cudaStreamWaitEvent(st, p->ev_tengy[h], 0));
    return TRPDRV_OK;
}

/* Emulated form: slice every operand once per execution, then per batch of `batch` triples (in the
 * processing order) one contraction launch writing their f and one energy launch on the second stream. */
static int enqueue_emulated(trpdrv_plan *p, cudaStream_t st, int capturing)
{
    int64_t launches = 0, bi = 0;
    p->tengy_sent[0] = p->tengy_sent[1] = 0;
    CUDA_TRY(cudaMemsetAsync(p->d_status, 0, sizeof(int), st));
    CUDA_TRY(cudaEventRecordWithFlags(p->ev0, st, capturing ? cudaEventRecordExternal : cudaEventRecordDefault));
    for (int q = 0; q < p->nsys; ++q) {
        const trpdrv_dev_system *d = &p->h_dev[q];
        const sysbuf *b = &p->s[q];
        if (d->ntriples <= 0) continue;
        LAUNCH_TRY(trpdrv_launch_oz_slices(d, &b->oz, st));
        ++launches;
        TRY(emulated_batches(p, d, b, 0, d->ntriples, p->opt.batch, st, &bi, &launches));
    }
    TRY(emulated_join(p, st));
    CUDA_TRY(cudaEventRecordWithFlags(p->ev1, st, capturing ? cudaEventRecordExternal : cudaEventRecordDefault));
    TRY(enqueue_finish(p, st, &launches));
    p->last_launches = launches;
    return TRPDRV_OK;
}

static int enqueue_device(trpdrv_plan *p, cudaStream_t st, int capturing)
{
    return p->opt.mode == TRPDRV_MODE_EMULATED ? enqueue_emulated(p, st, capturing) : enqueue_fused(p, st, capturing);
}

static int enqueue_plain(trpdrv_plan *p, cudaStream_t st)
{
    int64_t launches = 0;
    CUDA_TRY(cudaEventRecord(p->ev0, st));
    for (int q = 0; q < p->nsys; ++q) {
        const sysbuf *b = &p->s[q];
        const int64_t batch = plain_batch(b, p->plain_cap);
        for (int64_t r = 0; r < b->ntriples; r += batch) {
            const int n = (int)(b->ntriples - r < batch ? b->ntriples - r : batch);
            LAUNCH_TRY(trpdrv_launch_plain_batch(&p->h_dev[q], r, n, p->d_f, p->d_bpart, p->d_tcount, p->vec2, r > 0, st));
            launches += 2;
        }
    }
    CUDA_TRY(cudaEventRecord(p->ev1, st));
    TRY(enqueue_finish(p, st, &launches));
    p->last_launches = launches;
    return TRPDRV_OK;
}

int trpdrv_plan_execute(trpdrv_plan *p, void *stream)
{
    if (!p) return fail(TRPDRV_ERR_ARG, "NULL plan");
    if (!p->bound) return fail(TRPDRV_ERR_STATE, "execute before upload/bind");
    CUDA_TRY(cudaSetDevice(p->device));
    cudaStream_t st = stream ? (cudaStream_t)stream : p->stream;
    p->last_stream = st;
    p->events_valid = 0;
    if (p->opt.mode == TRPDRV_MODE_PLAIN) {
        TRY(enqueue_plain(p, st));
    } else if (p->opt.use_graph) {
        if (!p->graph_ready) {
            CUDA_TRY(cudaStreamBeginCapture(p->stream, cudaStreamCaptureModeThreadLocal));
            const int rc = enqueue_device(p, p->stream, 1);
            cudaGraph_t g = NULL;
            const cudaError_t ce = cudaStreamEndCapture(p->stream, &g);
            if (rc != TRPDRV_OK) {
                if (g) cudaGraphDestroy(g);
                return rc;
            }
            CUDA_TRY(ce);
            p->graph = g;
            CUDA_TRY(cudaGraphInstantiate(&p->gexec, p->graph, 0));
            p->graph_ready = 1;
        }
        CUDA_TRY(cudaGraphLaunch(p->gexec, st));
    } else {
        TRY(enqueue_device(p, st, 0));
    }
    p->events_valid = 1;
    return TRPDRV_OK;
}

/* ------------------------------------------------------------------------------------------ */
/* upload overlapped with execution (fused form)                                                 */
/* ------------------------------------------------------------------------------------------ */

/* T2, JOV and KOV hold one block per j (T2[j][i], JOV[j][i], KOV[j][i]); a triple (i, j, k) reads
 * only block j of each.  Every other tensor is read by every j. */
static int tensor_j_blocked(int w) { return w == TRPDRV_T_T2 || w == TRPDRV_T_JOV || w == TRPDRV_T_KOV; }

/* j (0-based) of the triple at processing position t of system b. */
static int position_j(const sysbuf *b, int64_t t)
{
    const int32_t idx = b->h_order ? b->h_order[t] : (int32_t)t;
    return (b->h_triples[idx] >> 10) & 1023;
}

/* One launch of the fused kernel over work items [first, end) of system q, preceded (for the
 * positions [p0, p1) of the first a) by the copies of the j blocks they read first. */
typedef struct chunk_span {
    int q;
    int64_t p0, p1;
    int64_t first, end;
} chunk_span;

static int chunk_spans(const trpdrv_plan *p, int chunks, chunk_span **out, int *nout)
{
    int64_t cap = 0, maxnt = 1;
    for (int q = 0; q < p->nsys; ++q) {
        cap += chunks + 1;
        if (p->s[q].nt > maxnt) maxnt = p->s[q].nt;
    }
    chunk_span *sp = (chunk_span *)malloc(sizeof(chunk_span) * (size_t)cap);
    int32_t *ijk = (int32_t *)malloc(sizeof(int32_t) * 3 * (size_t)maxnt);
    int64_t *bounds = (int64_t *)malloc(sizeof(int64_t) * ((size_t)chunks + 1));
    if (!sp || !ijk || !bounds) {
        free(sp);
        free(ijk);
        free(bounds);
        return fail(TRPDRV_ERR_NOMEM, "host allocation failed");
    }
    int n = 0;
    for (int q = 0; q < p->nsys; ++q) {
        const sysbuf *b = &p->s[q];
        const trpdrv_dev_system *d = &p->h_dev[q];
        const int64_t nt = b->nt, np = b->npairs;
        for (int64_t t = 0; t < nt; ++t) {
            const int pk = b->h_triples[t];
            ijk[3 * t] = (pk & 1023) + 1;
            ijk[3 * t + 1] = ((pk >> 10) & 1023) + 1;
            ijk[3 * t + 2] = ((pk >> 20) & 1023) + 1;
        }
        /* the first a's positions; the other a values read blocks that are all resident by then */
        const int64_t ns = trpdrv_upload_spans(ijk, b->h_order, nt, chunks, bounds);
        if (ns < 0) {
            free(sp);
            free(ijk);
            free(bounds);
            return fail(TRPDRV_ERR_ARG, "system %d: cannot split the processing order", q);
        }
        for (int64_t c = 0; c < ns; ++c)
            sp[n++] = (chunk_span){q, bounds[c], bounds[c + 1], d->item_begin + bounds[c] * np,
                                   d->item_begin + bounds[c + 1] * np};
        if (b->n_a > 1 && nt > 0)
            sp[n++] = (chunk_span){q, -1, -1, d->item_begin + nt * np, d->item_begin + b->ntriples * np};
    }
    free(ijk);
    free(bounds);
    *out = sp;
    *nout = n;
    return TRPDRV_OK;
}

static int span_resources(trpdrv_plan *p, int n)
{
    if (!p->copy_stream) CUDA_TRY(cudaStreamCreateWithFlags(&p->copy_stream, cudaStreamNonBlocking));
    if (!p->ev_in) CUDA_TRY(cudaEventCreateWithFlags(&p->ev_in, cudaEventDisableTiming));
    if (!p->ev_out) CUDA_TRY(cudaEventCreateWithFlags(&p->ev_out, cudaEventDisableTiming));
    if (n > p->nchunk_ev) {
        cudaEvent_t *ev = (cudaEvent_t *)realloc(p->chunk_ev, sizeof(cudaEvent_t) * (size_t)n);
        if (!ev) return fail(TRPDRV_ERR_NOMEM, "host allocation failed");
        p->chunk_ev = ev;
        while (p->nchunk_ev < n) {
            CUDA_TRY(cudaEventCreateWithFlags(&p->chunk_ev[p->nchunk_ev], cudaEventDisableTiming));
            ++p->nchunk_ev;
        }
    }
    if (n > p->nchunk_first) {
        if (p->d_chunk_first) cudaFree(p->d_chunk_first);
        free(p->h_chunk_first);
        p->d_chunk_first = NULL;
        p->nchunk_first = 0;
        p->h_chunk_first = (unsigned long long *)malloc(sizeof(unsigned long long) * (size_t)n);
        if (!p->h_chunk_first) return fail(TRPDRV_ERR_NOMEM, "host allocation failed");
        CUDA_TRY(cudaMalloc((void **)&p->d_chunk_first, sizeof(unsigned long long) * (size_t)n));
        p->nchunk_first = n;
    }
    return TRPDRV_OK;
}

/* Copies blocks j = lo .. hi-1 of T2, JOV and KOV of system q on the copy stream. */
static int copy_j_blocks(trpdrv_plan *p, const trpdrv_system *host, int q, int lo, int hi)
{
    const sysbuf *b = &p->s[q];
    for (int w = 0; w < TRPDRV_T_COUNT; ++w) {
        if (!tensor_j_blocked(w)) continue;
        const size_t blk = upload_elems(b, w) / (size_t)b->shape.nocc;
        CUDA_TRY(cudaMemcpyAsync(b->own[w] + (size_t)lo * blk, sys_tensor(&host[q], w) + (size_t)lo * blk,
                                 sizeof(double) * blk * (size_t)(hi - lo), cudaMemcpyHostToDevice, p->copy_stream));
    }
    return TRPDRV_OK;
}

/* Copies the j blocks that positions [p0, p1) of the span's system read and no earlier span of it
 * copied (have[j] marks the copied ones), one copy per run of consecutive j. */
static int span_copies(trpdrv_plan *p, const trpdrv_system *host, const chunk_span *c, unsigned char *have)
{
    const sysbuf *b = &p->s[c->q];
    int lo = -1, hi = -1;
    for (int64_t t = c->p0; t < c->p1; ++t) {
        const int j = position_j(b, t);
        if (have[j]) continue;
        have[j] = 1;
        if (j == hi) {
            ++hi;
            continue;
        }
        if (lo >= 0) TRY(copy_j_blocks(p, host, c->q, lo, hi));
        lo = j;
        hi = j + 1;
    }
    if (lo >= 0) TRY(copy_j_blocks(p, host, c->q, lo, hi));
    return TRPDRV_OK;
}

int trpdrv_plan_upload_execute(trpdrv_plan *p, const trpdrv_system *host, int chunks, void *stream)
{
    if (!p || !host) return fail(TRPDRV_ERR_ARG, "NULL plan or systems");
    if (chunks < 0 || chunks > 4096) return fail(TRPDRV_ERR_ARG, "chunks %d: must be 0..4096", chunks);
    if (p->opt.mode != TRPDRV_MODE_FUSED) { /* every digit slice needs all of T2 first */
        TRY(trpdrv_plan_upload(p, host, stream));
        return trpdrv_plan_execute(p, stream);
    }
    if (chunks == 0) chunks = 16;
    CUDA_TRY(cudaSetDevice(p->device));
    cudaStream_t user = stream ? (cudaStream_t)stream : NULL;
    TRY(upload_prepare(p, host));
    chunk_span *sp = NULL;
    int nsp = 0;
    TRY(chunk_spans(p, chunks, &sp, &nsp));
    int rc = span_resources(p, nsp > 0 ? nsp : 1);
    unsigned char *have = NULL;
    int maxo = 1;
    for (int q = 0; q < p->nsys; ++q)
        if (p->s[q].shape.nocc > maxo) maxo = p->s[q].shape.nocc;
    if (rc == TRPDRV_OK && !(have = (unsigned char *)malloc(2 * (size_t)maxo)))
        rc = fail(TRPDRV_ERR_NOMEM, "host allocation failed");
#define STEP(call)                          \
    do {                                    \
        if (rc == TRPDRV_OK) rc = (call);   \
    } while (0)
#define STEP_CUDA(call)                                                                             \
    do {                                                                                            \
        if (rc == TRPDRV_OK) {                                                                      \
            cudaError_t e_ = (call);                                                                \
            if (e_ != cudaSuccess) {                                                                \
                cudaGetLastError();                                                                 \
                rc = fail(TRPDRV_ERR_CUDA, "%s: %s (%s:%d)", #call, cudaGetErrorString(e_), __FILE__, __LINE__); \
            }                                                                                       \
        }                                                                                           \
    } while (0)
    /* both streams after the caller's stream and after the previous execution */
    if (user) {
        STEP_CUDA(cudaEventRecord(p->ev_in, user));
        STEP_CUDA(cudaStreamWaitEvent(p->stream, p->ev_in, 0));
    }
    if (p->last_stream && p->last_stream != p->stream && p->last_stream != user) {
        STEP_CUDA(cudaEventRecord(p->ev_in, p->last_stream));
        STEP_CUDA(cudaStreamWaitEvent(p->stream, p->ev_in, 0));
    }
    STEP_CUDA(cudaEventRecord(p->ev_in, p->stream));
    STEP_CUDA(cudaStreamWaitEvent(p->copy_stream, p->ev_in, 0));
    /* the tensors every j reads, then the plan's derived arrays and tensor maps */
    for (int q = 0; q < p->nsys && rc == TRPDRV_OK; ++q)
        for (int w = 0; w < TRPDRV_T_COUNT; ++w)
            if (!tensor_j_blocked(w))
                STEP_CUDA(cudaMemcpyAsync(p->s[q].own[w], sys_tensor(&host[q], w),
                                          sizeof(double) * upload_elems(&p->s[q], w), cudaMemcpyHostToDevice,
                                          p->stream));
    STEP(plan_publish(p));
    /* per span: its j blocks on the copy stream, then the kernel over its items once they are in */
    if (rc == TRPDRV_OK)
        for (int c = 0; c < nsp; ++c) p->h_chunk_first[c] = (unsigned long long)sp[c].first;
    STEP_CUDA(cudaMemsetAsync(p->d_status, 0, sizeof(int), p->stream));
    if (nsp > 0)
        STEP_CUDA(cudaMemcpyAsync(p->d_chunk_first, p->h_chunk_first, sizeof(unsigned long long) * (size_t)nsp,
                                  cudaMemcpyHostToDevice, p->stream));
    STEP_CUDA(cudaEventRecord(p->ev0, p->stream));
    int64_t launches = 0;
    int prev_q = -1;
    for (int c = 0; c < nsp && rc == TRPDRV_OK; ++c) {
        if (sp[c].q != prev_q) {
            memset(have, 0, 2 * (size_t)maxo);
            prev_q = sp[c].q;
            STEP(pad_refill(p, sp[c].q, 1, 0, 0, p->stream, &launches));
        }
        if (sp[c].p0 >= 0) {
            unsigned char *padded = have + maxo; /* j blocks already in the padded copies */
            STEP(span_copies(p, host, &sp[c], have));
            STEP_CUDA(cudaEventRecord(p->chunk_ev[c], p->copy_stream));
            STEP_CUDA(cudaStreamWaitEvent(p->stream, p->chunk_ev[c], 0));
            for (int lo = 0; lo < p->s[sp[c].q].shape.nocc;) {
                int hi = lo;
                while (hi < p->s[sp[c].q].shape.nocc && have[hi] && !padded[hi]) padded[hi++] = 1;
                if (hi > lo) STEP(pad_refill(p, sp[c].q, 0, lo, hi, p->stream, &launches));
                lo = hi > lo ? hi : lo + 1;
            }
        }
        const int64_t n = sp[c].end - sp[c].first;
        const int cap = p->use_tma ? p->grid_tma : p->grid;
        const int grid = (int64_t)cap < n ? cap : (int)n;
        if (n <= 0 || rc != TRPDRV_OK) continue;
        int e = p->use_tma ? trpdrv_launch_fused_tma(p->d_dev, p->nsys, sp[c].end, 0, p->d_chunk_first + c, p->d_status,
                                                     grid, p->tma_maps, p->tma_mma_k, p->stream)
                           : trpdrv_launch_fused(p->d_dev, p->nsys, sp[c].end, 0, p->d_chunk_first + c, p->d_status,
                                                 grid, p->vec2 || p->padded, p->opt.mma_k, p->stream);
        if (e) rc = fail(TRPDRV_ERR_CUDA, "fused launch of span %d: %s", c, cudaGetErrorString((cudaError_t)e));
        ++launches;
    }
    STEP_CUDA(cudaEventRecord(p->ev1, p->stream));
    STEP(enqueue_finish(p, p->stream, &launches));
    if (user) {
        STEP_CUDA(cudaEventRecord(p->ev_out, p->stream));
        STEP_CUDA(cudaStreamWaitEvent(user, p->ev_out, 0));
    }
#undef STEP
#undef STEP_CUDA
    free(have);
    free(sp);
    if (rc != TRPDRV_OK) return rc;
    p->last_launches = launches;
    p->last_stream = user ? user : p->stream;
    p->events_valid = 1;
    return TRPDRV_OK;
}

static int plan_wait(trpdrv_plan *p)
{
    CUDA_TRY(cudaSetDevice(p->device));
    CUDA_TRY(cudaStreamSynchronize(p->last_stream ? p->last_stream : p->stream));
    p->last_stream = NULL; /* the job is done: the caller may now destroy its stream */
    const int status = (int)p->h_res[4 * p->nsys];
    if (status & 2) return fail(TRPDRV_ERR_DEVICE, "a fused-kernel pipeline wait ran out of time");
    if (status) return fail(TRPDRV_ERR_DEVICE, "a device kernel rejected a malformed work-queue entry");
    return TRPDRV_OK;
}

int trpdrv_plan_energies(trpdrv_plan *p, double *emp4, double *emp5)
{
    if (!p) return fail(TRPDRV_ERR_ARG, "NULL plan");
    TRY(plan_wait(p));
    for (int q = 0; q < p->nsys; ++q) {
        const double *tot = p->h_res + 4 * q;
        if (emp4) emp4[q] = tot[0] + tot[1];
        if (emp5) emp5[q] = tot[2] + tot[3];
    }
    return TRPDRV_OK;
}

int64_t trpdrv_plan_num_triples(const trpdrv_plan *p, int sys)
{
    if (!p || sys < 0 || sys >= p->nsys) return -1;
    return p->s[sys].ntriples;
}

int trpdrv_plan_triples(const trpdrv_plan *p, int sys, int32_t *ijk)
{
    if (!p || sys < 0 || sys >= p->nsys || !ijk) return fail(TRPDRV_ERR_ARG, "bad plan/sys/output");
    const sysbuf *b = &p->s[sys];
    for (int64_t t = 0; t < b->ntriples; ++t) {
        const int pk = b->h_triples[t % b->nt]; /* records are [a][triple] */
        ijk[3 * t + 0] = (pk & 1023) + 1;
        ijk[3 * t + 1] = ((pk >> 10) & 1023) + 1;
        ijk[3 * t + 2] = ((pk >> 20) & 1023) + 1;
    }
    return TRPDRV_OK;
}

int trpdrv_plan_triple_energies(trpdrv_plan *p, int sys, double *rec)
{
    if (!p || sys < 0 || sys >= p->nsys || !rec) return fail(TRPDRV_ERR_ARG, "bad plan/sys/output");
    TRY(plan_wait(p));
    const sysbuf *b = &p->s[sys];
    if (b->ntriples > 0)
        CUDA_TRY(cudaMemcpy(rec, b->rec, sizeof(double) * 4 * (size_t)b->ntriples, cudaMemcpyDeviceToHost));
    return TRPDRV_OK;
}

int64_t trpdrv_plan_last_launches(const trpdrv_plan *p) { return p ? p->last_launches : -1; }

int trpdrv_plan_staging(const trpdrv_plan *p)
{
    if (!p || !p->bound || p->opt.mode != TRPDRV_MODE_FUSED) return 0;
    return p->use_tma ? 2 : 1;
}

int trpdrv_plan_last_kernel_ms(trpdrv_plan *p, double *ms)
{
    if (!p || !ms) return fail(TRPDRV_ERR_ARG, "NULL plan/output");
    if (!p->events_valid) return fail(TRPDRV_ERR_STATE, "no execute to time");
    TRY(plan_wait(p));
    float f = 0.0f;
    CUDA_TRY(cudaEventElapsedTime(&f, p->ev0, p->ev1));
    *ms = (double)f;
    return TRPDRV_OK;
}

/* ------------------------------------------------------------------------------------------ */
/* autotuner                                                                                    */
/* ------------------------------------------------------------------------------------------ */

typedef struct tune_entry {
    int used, dev, mode, slices, world, rank, nsys, staging, a_count;
    int shape[3 * TRPDRV_TMA_MAX_SYSTEMS];
    trpdrv_tune_candidate best;
} tune_entry;

static tune_entry g_tune[64];
static pthread_mutex_t g_tune_mu = PTHREAD_MUTEX_INITIALIZER;

static void tune_key(const trpdrv_plan *p, tune_entry *k)
{
    memset(k, 0, sizeof *k);
    k->dev = p->device;
    k->mode = p->opt.mode;
    k->slices = p->opt.mode == TRPDRV_MODE_EMULATED ? p->opt.slices : 0;
    k->world = p->opt.world;
    k->rank = p->opt.rank;
    k->nsys = p->nsys;
    k->staging = p->opt.staging; /* a forced staging limits the candidates */
    k->a_count = p->opt.a_count;
    for (int q = 0; q < p->nsys && q < TRPDRV_TMA_MAX_SYSTEMS; ++q) {
        k->shape[3 * q] = p->s[q].shape.nocc;
        k->shape[3 * q + 1] = p->s[q].shape.nvir;
        k->shape[3 * q + 2] = p->opt.nkpass;
    }
}

static int tune_same(const tune_entry *a, const tune_entry *b)
{
    return a->dev == b->dev && a->mode == b->mode && a->slices == b->slices && a->world == b->world &&
           a->rank == b->rank && a->nsys == b->nsys && a->staging == b->staging && a->a_count == b->a_count &&
           memcmp(a->shape, b->shape, sizeof a->shape) == 0;
}

/* ---- persistent tuning cache (TRPDRV_TUNE_CACHE = path of a text file shared by processes) ----
 * One line per choice: "<key> -> <staging> <mma_k> <ctas_per_sm> <batch> <edge_pack> <ms>", where the key names
 * the device model (name, SM count), the library version, the revision of the kernels and every field of tune_entry.  Lookups
 * take the last matching line; stores append under an exclusive lock. */
/* Raised whenever the kernels that candidates are timed with change: choices made with others are timed again. */
#define TUNE_KERNELS 2
static int tune_file_key(const trpdrv_plan *p, const tune_entry *k, char *buf, size_t n)
{
    struct cudaDeviceProp prop;
    if (cudaGetDeviceProperties(&prop, p->device) != cudaSuccess) return -1;
    char name[96];
    size_t q = 0;
    for (const char *c = prop.name; *c && q + 1 < sizeof name; ++c) name[q++] = (*c == ' ' || *c == '>') ? '_' : *c;
    name[q] = '\0';
    int w = snprintf(buf, n, "trpdrv-tune v%d.%d %s sm%d mode=%d slices=%d world=%d rank=%d staging=%d a=%d nsys=%d shapes=",
                     trpdrv_version(), TUNE_KERNELS, name, prop.multiProcessorCount, k->mode, k->slices, k->world, k->rank,
                     k->staging, k->a_count, k->nsys);
    for (int s = 0; s < k->nsys && s < TRPDRV_TMA_MAX_SYSTEMS && w > 0 && (size_t)w < n; ++s)
        w += snprintf(buf + w, n - (size_t)w, "%s%d,%d,%d", s ? ";" : "", k->shape[3 * s], k->shape[3 * s + 1],
                      k->shape[3 * s + 2]);
    return (w > 0 && (size_t)w < n) ? 0 : -1;
}

static int tune_file_lookup(const char *key, trpdrv_tune_candidate *out)
{
    const char *path = getenv("TRPDRV_TUNE_CACHE");
    if (!path || !*path) return 0;
    FILE *f = fopen(path, "r");
    if (!f) return 0;
    flock(fileno(f), LOCK_SH);
    char line[1024];
    const size_t kl = strlen(key);
    int found = 0;
    while (fgets(line, sizeof line, f)) {
        if (strncmp(line, key, kl) != 0 || strncmp(line + kl, " -> ", 4) != 0) continue;
        trpdrv_tune_candidate c;
        memset(&c, 0, sizeof c);
        if (sscanf(line + kl + 4, "%d %d %d %d %d %lf", &c.staging, &c.mma_k, &c.ctas_per_sm, &c.batch, &c.edge_pack,
                   &c.ms_estimate) == 6) {
            *out = c;
            found = 1;
        }
    }
    flock(fileno(f), LOCK_UN);
    fclose(f);
    return found;
}

static void tune_file_store(const char *key, const trpdrv_tune_candidate *c)
{
    const char *path = getenv("TRPDRV_TUNE_CACHE");
    if (!path || !*path) return;
    const int fd = open(path, O_WRONLY | O_APPEND | O_CREAT, 0644);
    if (fd < 0) return;
    char line[1200];
    const int n = snprintf(line, sizeof line, "%s -> %d %d %d %d %d %.6f\n", key, c->staging, c->mma_k,
                           c->ctas_per_sm, c->batch, c->edge_pack, c->ms_estimate);
    if (n > 0 && (size_t)n < sizeof line && flock(fd, LOCK_EX) == 0) {
        ssize_t wr = write(fd, line, (size_t)n);
        (void)wr;
        flock(fd, LOCK_UN);
    }
    close(fd);
}

/* a cached choice is usable only if this plan can run it */
static int tune_usable(const trpdrv_plan *p, const trpdrv_tune_candidate *c)
{
    if (p->opt.mode == TRPDRV_MODE_FUSED) {
        if (c->staging == 2)
            return p->opt.staging != 1 && p->tma_maps && trpdrv_tma_supported(p->h_dev, p->nsys) &&
                   (c->mma_k == 8 || c->mma_k == 16);
        return c->staging == 1 && p->opt.staging != 2 && (c->mma_k == 4 || c->mma_k == 8) && c->ctas_per_sm >= 1;
    }
    return c->batch >= 1 && c->batch <= p->fbuf_batch;
}

/* the fused kernel's edge tile shape on every system (host mirror and device copy of the descriptors) */
static int tune_set_edge_pack(trpdrv_plan *p, int pack)
{
    int changed = 0;
    for (int q = 0; q < p->nsys; ++q) {
        const int v = pack ? trpdrv_tma_pack_edge(p->s[q].shape.nvir) : 0;
        changed |= p->h_dev[q].pack_edge != v;
        p->h_dev[q].pack_edge = v;
    }
    if (changed && p->d_dev)
        CUDA_TRY(cudaMemcpy(p->d_dev, p->h_dev, sizeof(trpdrv_dev_system) * (size_t)p->nsys, cudaMemcpyHostToDevice));
    return TRPDRV_OK;
}

/* sets the plan's launch configuration to candidate c */
static void tune_apply(trpdrv_plan *p, const trpdrv_tune_candidate *c)
{
    if (p->opt.mode == TRPDRV_MODE_FUSED) {
        p->use_tma = c->staging == 2;
        p->tuned_staging = c->staging; /* a later upload/bind keeps it where TMA remains possible */
        if (c->staging == 2) p->tma_mma_k = c->mma_k;
        tune_set_edge_pack(p, c->edge_pack);
        if (c->staging == 1) {
            p->opt.mma_k = c->mma_k;
            p->opt.ctas_per_sm = c->ctas_per_sm;
            int64_t grid = (int64_t)c->ctas_per_sm * p->nsm;
            if (grid > p->total_items) grid = p->total_items;
            p->grid = (int)(grid > 0 ? grid : 0);
        }
    } else if (p->opt.mode == TRPDRV_MODE_EMULATED) {
        p->opt.batch = c->batch;
    }
    if (p->graph_ready) {
        cudaGraphExecDestroy(p->gexec);
        cudaGraphDestroy(p->graph);
        p->gexec = NULL;
        p->graph = NULL;
        p->graph_ready = 0;
    }
}

static int tune_elapsed(trpdrv_plan *p, float *ms)
{
    CUDA_TRY(cudaEventSynchronize(p->ev1));
    CUDA_TRY(cudaEventElapsedTime(ms, p->ev0, p->ev1));
    return TRPDRV_OK;
}

/* estimated device time of one execution with candidate c: each system timed on a sample (the best of
 * TUNE_REPS runs of the same sample, the first of which also warms the caches) and scaled to its full
 * work; candidates within a few percent of each other need the minimum to be told apart */
#define TUNE_REPS 3
static int tune_time(trpdrv_plan *p, const trpdrv_tune_candidate *c, double *est)
{
    cudaStream_t st = p->stream;
    *est = 0.0;
    for (int q = 0; q < p->nsys; ++q) {
        const trpdrv_dev_system *d = &p->h_dev[q];
        if (d->ntriples <= 0) continue;
        float ms = 0.0f;
        if (p->opt.mode == TRPDRV_MODE_FUSED) {
            TRY(pad_refill(p, q, 1, 0, p->s[q].shape.nocc, st, NULL));
            const int64_t items = d->ntriples * d->npairs;
            int64_t sample = items / 8;
            if (sample < (int64_t)p->nsm * 64) sample = (int64_t)p->nsm * 64;
            if (sample > items) sample = items;
            const unsigned long long first = (unsigned long long)d->item_begin;
            int grid = c->staging == 2 ? p->nsm : c->ctas_per_sm * p->nsm;
            if (grid > sample) grid = (int)sample;
            TRY(tune_set_edge_pack(p, c->edge_pack));
            /* in the order in which the plan runs them; plans that run pair by pair are timed whole */
            const int pair_major = plan_pair_major(p) && sample == items;
            float best = 0.0f;
            for (int rep = 0; rep < TUNE_REPS; ++rep) {
                CUDA_TRY(cudaMemcpyAsync(p->d_counter, &first, sizeof first, cudaMemcpyHostToDevice, st));
                CUDA_TRY(cudaStreamSynchronize(st)); /* `first` is a host stack value */
                CUDA_TRY(cudaEventRecord(p->ev0, st));
                if (c->staging == 2)
                    LAUNCH_TRY(trpdrv_launch_fused_tma(p->d_dev, p->nsys, d->item_begin + sample, pair_major, p->d_counter,
                                                       p->d_status, grid, p->tma_maps, c->mma_k, st));
                else
                    LAUNCH_TRY(trpdrv_launch_fused(p->d_dev, p->nsys, d->item_begin + sample, pair_major, p->d_counter,
                                                   p->d_status, grid, p->vec2 || p->padded, c->mma_k, st));
                CUDA_TRY(cudaEventRecord(p->ev1, st));
                TRY(tune_elapsed(p, &ms));
                if (rep == 0 || ms < best) best = ms;
            }
            *est += (double)best * (double)items / (double)sample;
        } else {
            const sysbuf *b = &p->s[q];
            /* four launch pairs of the largest batch, so every candidate is timed over several launches */
            const int64_t want = 4 * (int64_t)TUNE_MAX_BATCH;
            const int64_t n = d->ntriples < want ? d->ntriples : want;
            LAUNCH_TRY(trpdrv_launch_oz_slices(d, &b->oz, st));
            float best = 0.0f;
            for (int rep = 0; rep < TUNE_REPS; ++rep) {
                int64_t bi = 0;
                CUDA_TRY(cudaEventRecord(p->ev0, st));
                TRY(emulated_batches(p, d, b, 0, n, c->batch, st, &bi, NULL));
                TRY(emulated_join(p, st));
                CUDA_TRY(cudaEventRecord(p->ev1, st));
                TRY(tune_elapsed(p, &ms));
                if (rep == 0 || ms < best) best = ms;
            }
            *est += (double)best * (double)d->ntriples / (double)n;
        }
    }
    return TRPDRV_OK;
}

/* emulated plans: switch every system to `slices` digit slices (the buffers hold 8) */
static int tune_set_slices(trpdrv_plan *p, int slices)
{
    for (int q = 0; q < p->nsys; ++q) {
        p->s[q].oz.slices = slices;
        const int e = trpdrv_oz_prepare(&p->s[q].oz, p->s[q].oz_maps);
        if (e) return fail(TRPDRV_ERR_CUDA, "tensor-map encoding failed (%d)", e);
    }
    p->opt.slices = slices;
    if (p->graph_ready) {
        cudaGraphExecDestroy(p->gexec);
        cudaGraphDestroy(p->graph);
        p->gexec = NULL;
        p->graph = NULL;
        p->graph_ready = 0;
    }
    return TRPDRV_OK;
}

/* emulated plans: per-triple records of the first 64 positions of every system (the other records keep
 * what they held), copied to host[q] (ntriples * 4 each) */
static int tune_sample_records(trpdrv_plan *p, double **host)
{
    cudaStream_t st = p->stream;
    for (int q = 0; q < p->nsys; ++q) {
        const trpdrv_dev_system *d = &p->h_dev[q];
        const sysbuf *b = &p->s[q];
        if (d->ntriples <= 0) continue;
        const int64_t n = d->ntriples < 64 ? d->ntriples : 64;
        LAUNCH_TRY(trpdrv_launch_oz_slices(d, &b->oz, st));
        int64_t bi = 0;
        TRY(emulated_batches(p, d, b, 0, n, p->opt.batch, st, &bi, NULL));
        TRY(emulated_join(p, st));
    }
    /* the records alone: the totals stay those of the last execution */
    LAUNCH_TRY(trpdrv_launch_records(p->h_dev, p->d_dev, p->nsys, st));
    for (int q = 0; q < p->nsys; ++q)
        if (p->s[q].ntriples > 0)
            CUDA_TRY(cudaMemcpyAsync(host[q], p->s[q].rec, sizeof(double) * 4 * (size_t)p->s[q].ntriples,
                                     cudaMemcpyDeviceToHost, st));
    CUDA_TRY(cudaStreamSynchronize(st));
    return TRPDRV_OK;
}

/* largest normwise (per energy column) deviation of got from want over every system's records */
static double tune_record_dev(const trpdrv_plan *p, double **got, double **want)
{
    double worst = 0.0;
    for (int q = 0; q < p->nsys; ++q)
        for (int c = 0; c < 4; ++c) {
            double scale = 0.0, dev = 0.0;
            for (int64_t t = 0; t < p->s[q].ntriples; ++t) {
                const double w = fabs(want[q][4 * t + c]), e = fabs(got[q][4 * t + c] - want[q][4 * t + c]);
                if (w > scale) scale = w;
                if (e > dev) dev = e;
            }
            if (scale > 0.0 && dev / scale > worst) worst = dev / scale;
        }
    return worst;
}

/* emulated plans with target_digits: the fewest slices (4..7, else 8) whose sampled records agree with
 * those of 8 slices to a tenth of the target */
static int tune_choose_slices(trpdrv_plan *p, double *est)
{
    const double target = pow(10.0, -(double)(p->opt.target_digits + 1));
    double **ref = (double **)calloc((size_t)p->nsys, sizeof(double *));
    double **got = (double **)calloc((size_t)p->nsys, sizeof(double *));
    int rc = (ref && got) ? TRPDRV_OK : fail(TRPDRV_ERR_NOMEM, "host allocation failed");
    for (int q = 0; q < p->nsys && rc == TRPDRV_OK; ++q) {
        const size_t n = 4 * (size_t)(p->s[q].ntriples > 0 ? p->s[q].ntriples : 1);
        ref[q] = (double *)calloc(n, sizeof(double));
        got[q] = (double *)calloc(n, sizeof(double));
        if (!ref[q] || !got[q]) rc = fail(TRPDRV_ERR_NOMEM, "host allocation failed");
    }
    int chosen = 8;
    double dev = 0.0, prev = 0.0;
    if (rc == TRPDRV_OK) rc = tune_set_slices(p, 8);
    if (rc == TRPDRV_OK) rc = tune_sample_records(p, ref);
    for (int sl = TRPDRV_OZ_MIN_SLICES; sl < 8 && rc == TRPDRV_OK; ++sl) {
        rc = tune_set_slices(p, sl);
        if (rc == TRPDRV_OK) rc = tune_sample_records(p, got);
        if (rc != TRPDRV_OK) break;
        dev = tune_record_dev(p, got, ref);
        prev = dev;
        if (dev <= target) {
            chosen = sl;
            break;
        }
    }
    if (rc == TRPDRV_OK) {
        rc = tune_set_slices(p, chosen);
        /* 8 slices: its own deviation is about 2^-7 of 7 slices' */
        *est = chosen == 8 ? prev / 128.0 : dev;
    }
    for (int q = 0; q < p->nsys; ++q) {
        if (ref) free(ref[q]);
        if (got) free(got[q]);
    }
    free(ref);
    free(got);
    return rc;
}

int trpdrv_plan_autotune(trpdrv_plan *p, trpdrv_tune_result *result)
{
    trpdrv_tune_result local;
    trpdrv_tune_result *r = result ? result : &local;
    memset(r, 0, sizeof *r);
    if (!p) return fail(TRPDRV_ERR_ARG, "NULL plan");
    if (!p->bound) return fail(TRPDRV_ERR_STATE, "autotune before upload/bind");
    if (p->opt.mode == TRPDRV_MODE_PLAIN) return TRPDRV_OK; /* one compiled form: nothing to choose */
    CUDA_TRY(cudaSetDevice(p->device));
    p->events_valid = 0; /* the timing below reuses the plan's events */

    double est = 0.0;
    if (p->opt.mode == TRPDRV_MODE_EMULATED && p->opt.target_digits > 0) {
        CUDA_TRY(cudaMemsetAsync(p->d_status, 0, sizeof(int), p->stream));
        TRY(tune_choose_slices(p, &est));
    }
    r->slices = p->opt.mode == TRPDRV_MODE_EMULATED ? p->opt.slices : 0;
    r->est_rel_err = est;

    tune_entry key;
    tune_key(p, &key);
    const int cacheable = p->nsys <= TRPDRV_TMA_MAX_SYSTEMS && p->opt.target_digits == 0;
    if (cacheable) {
        pthread_mutex_lock(&g_tune_mu);
        int hit = -1;
        for (int e = 0; e < (int)(sizeof g_tune / sizeof g_tune[0]); ++e)
            if (g_tune[e].used && tune_same(&g_tune[e], &key)) hit = e;
        trpdrv_tune_candidate best;
        memset(&best, 0, sizeof best);
        if (hit >= 0) best = g_tune[hit].best;
        pthread_mutex_unlock(&g_tune_mu);
        /* a cached choice applies only where this plan can run it */
        if (hit >= 0 && !tune_usable(p, &best)) hit = -1;
        if (hit >= 0) {
            r->ncand = 1;
            r->chosen = 0;
            r->from_cache = 1;
            r->cand[0] = best;
            tune_apply(p, &best);
            return TRPDRV_OK;
        }
        char fkey[768];
        if (tune_file_key(p, &key, fkey, sizeof fkey) == 0 && tune_file_lookup(fkey, &best) && tune_usable(p, &best)) {
            r->ncand = 1;
            r->chosen = 0;
            r->from_cache = 2;
            r->cand[0] = best;
            tune_apply(p, &best);
            pthread_mutex_lock(&g_tune_mu);
            int slot = -1;
            for (int e = 0; e < (int)(sizeof g_tune / sizeof g_tune[0]) && slot < 0; ++e)
                if (!g_tune[e].used) slot = e;
            if (slot < 0) slot = 0;
            g_tune[slot] = key;
            g_tune[slot].used = 1;
            g_tune[slot].best = best;
            pthread_mutex_unlock(&g_tune_mu);
            return TRPDRV_OK;
        }
    }

    /* candidates */
    trpdrv_tune_candidate *c = r->cand;
    int n = 0;
    if (p->opt.mode == TRPDRV_MODE_FUSED) {
        int packable = 0;
        for (int q = 0; q < p->nsys; ++q) packable |= trpdrv_tma_pack_edge(p->s[q].shape.nvir);
        if (p->opt.staging != 1 && trpdrv_tma_supported(p->h_dev, p->nsys) && p->tma_maps) {
            c[n++] = (trpdrv_tune_candidate){2, 8, 1, 0, packable, 0.0};
            c[n++] = (trpdrv_tune_candidate){2, 16, 1, 0, packable, 0.0};
            if (packable) {
                c[n++] = (trpdrv_tune_candidate){2, 8, 1, 0, 0, 0.0};
                c[n++] = (trpdrv_tune_candidate){2, 16, 1, 0, 0, 0.0};
            }
        }
        if (p->opt.staging != 2) {
            c[n++] = (trpdrv_tune_candidate){1, 8, 1, 0, packable, 0.0};
            c[n++] = (trpdrv_tune_candidate){1, 4, 1, 0, packable, 0.0};
        }
    } else {
        static const int batches[4] = {8, 16, 32, 64};
        for (int k = 0; k < 4; ++k)
            if (batches[k] <= p->fbuf_batch) c[n++] = (trpdrv_tune_candidate){0, 0, 0, batches[k], 0, 0.0};
    }
    r->ncand = n;
    if (n == 0) return TRPDRV_OK;

    CUDA_TRY(cudaMemsetAsync(p->d_status, 0, sizeof(int), p->stream));
    int best = 0;
    for (int k = 0; k < n; ++k) {
        TRY(tune_time(p, &c[k], &c[k].ms_estimate));
        if (c[k].ms_estimate < c[best].ms_estimate) best = k;
    }
    int status = 0;
    CUDA_TRY(cudaMemcpy(&status, p->d_status, sizeof(int), cudaMemcpyDeviceToHost));
    if (status) return fail(TRPDRV_ERR_DEVICE, "a device kernel reported status %d while autotuning", status);
    r->chosen = best;
    tune_apply(p, &c[best]);
    if (cacheable) {
        pthread_mutex_lock(&g_tune_mu);
        int slot = -1;
        for (int e = 0; e < (int)(sizeof g_tune / sizeof g_tune[0]) && slot < 0; ++e)
            if (!g_tune[e].used) slot = e;
        if (slot < 0) slot = 0; /* full: overwrite the oldest slot */
        g_tune[slot] = key;
        g_tune[slot].used = 1;
        g_tune[slot].best = c[best];
        pthread_mutex_unlock(&g_tune_mu);
        char fkey[768];
        if (tune_file_key(p, &key, fkey, sizeof fkey) == 0) tune_file_store(fkey, &c[best]);
    }
    return TRPDRV_OK;
}

int trpdrv_plan_destroy(trpdrv_plan *p)
{
    if (!p) return TRPDRV_OK;
    cudaSetDevice(p->device);
    cudaStreamSynchronize(p->stream);
    plan_free(p);
    return TRPDRV_OK;
}

int trpdrv_run(const trpdrv_system *host, int nsys, const trpdrv_options *opt, double *emp4, double *emp5)
{
    trpdrv_plan *p = NULL;
    TRY(trpdrv_plan_create(&p, host, nsys, opt));
    int rc = trpdrv_plan_upload_execute(p, host, 0, NULL);
    if (rc == TRPDRV_OK) rc = trpdrv_plan_energies(p, emp4, emp5);
    trpdrv_plan_destroy(p);
    return rc;
}

/* ------------------------------------------------------------------------------------------ */
/* drop-in entry points                                                                         */
/* ------------------------------------------------------------------------------------------ */

/* One triple's inputs as the drop-in body stages them, on the device and in a pinned host mirror (the two always
 * hold the same bytes once the transfers of a call have run):
 *   I    the i-role blocks: tij, jia, kia, tia, xia, jij, kij
 *   K    the k-role blocks: tkj, jka, kka, tka, xka, jkj, kkj
 *   VEC  dintc1, dintx1, t1v1, dintc2, dintx2, t1v2, eorb
 * Rows of odd length are padded to the next even one (zero pads), so that the GEMM copies 16 bytes at a time
 * whatever the sizes.  K and VEC, which the reference driver's k-inner loop (omp/test.c:160-176) changes from
 * call to call, are contiguous: a small call sends one piece. */
enum { DS_I = 0, DS_K = 7, DS_VEC = 14, DS_N = 21 };
enum { DS_T = 0, DS_J, DS_KV, DS_TO, DS_XO, DS_JO, DS_KO }; /* blocks of a role, after its first slot */

static struct dropin_state {
    int ready, device;
    cudaStream_t stream;
    int ncor, nocc, nvir;      /* shape of the staging layout */
    size_t off[DS_N + 1];      /* its slots' offsets (doubles) */
    size_t cap_stage;          /* doubles in d_stage / h_stage */
    double *d_stage, *h_stage;
    size_t cap_f, cap_part;
    double *f, *bpart;
    size_t cap_vec;
    double *vec;               /* the tengy entry points' vectors */
    unsigned *tcount;
    double *h_out4;            /* pinned: the energy kernel writes it directly */
} g_di;
static pthread_mutex_t g_di_mu = PTHREAD_MUTEX_INITIALIZER;

static int env_flag(const char *name, const char *value)
{
    const char *v = getenv(name);
    return v && strcmp(v, value) == 0;
}

/* Host arrays registered as unchanging (trpdrv_register_host): device copies that the drop-in entry
 * points read in place of per-call copies of any pointer inside them. */
#define DI_MAX_REG 64
static struct reg_entry {
    const char *host;
    size_t bytes;
    char *dev;
} g_reg[DI_MAX_REG];
static int g_nreg;

static void reg_release(void)
{
    for (int r = 0; r < g_nreg; ++r) cudaFree(g_reg[r].dev);
    memset(g_reg, 0, sizeof g_reg);
    g_nreg = 0;
}

/* device address of [p, p + n) if it lies inside a registered array, else NULL */
static const double *reg_lookup(const double *p, size_t n)
{
    const char *c = (const char *)p;
    for (int r = 0; r < g_nreg; ++r)
        if (c >= g_reg[r].host && c + n * sizeof(double) <= g_reg[r].host + g_reg[r].bytes)
            return (const double *)(g_reg[r].dev + (c - g_reg[r].host));
    return NULL;
}

static void di_release(void)
{
    if (!g_di.ready) return;
    cudaSetDevice(g_di.device);
    reg_release();
    cudaFree(g_di.d_stage);
    cudaFreeHost(g_di.h_stage);
    cudaFree(g_di.f);
    cudaFree(g_di.bpart);
    cudaFree(g_di.vec);
    cudaFree(g_di.tcount);
    cudaFreeHost(g_di.h_out4);
    cudaStreamDestroy(g_di.stream);
    memset(&g_di, 0, sizeof g_di);
}

static int di_reserve(int nocc, int nvir, int nbf);

int trpdrv_register_host(const void *ptr, size_t bytes)
{
    if (!ptr || bytes == 0) return fail(TRPDRV_ERR_ARG, "NULL pointer or empty range");
    pthread_mutex_lock(&g_di_mu);
    int rc = TRPDRV_OK;
    if (g_nreg >= DI_MAX_REG) {
        rc = fail(TRPDRV_ERR_ARG, "at most %d registered arrays", DI_MAX_REG);
    } else {
        const char *c = (const char *)ptr;
        for (int r = 0; r < g_nreg && rc == TRPDRV_OK; ++r)
            if (c < g_reg[r].host + g_reg[r].bytes && g_reg[r].host < c + bytes)
                rc = fail(TRPDRV_ERR_ARG, "range overlaps a registered array");
        if (rc == TRPDRV_OK) rc = di_reserve(1, 1, 1); /* device and stream of the drop-in entry points */
        char *dev = NULL;
        if (rc == TRPDRV_OK) {
            cudaError_t e = cudaMalloc((void **)&dev, bytes);
            if (e == cudaSuccess) e = cudaMemcpy(dev, ptr, bytes, cudaMemcpyHostToDevice);
            if (e != cudaSuccess) {
                cudaGetLastError();
                if (dev) cudaFree(dev);
                rc = fail(e == cudaErrorMemoryAllocation ? TRPDRV_ERR_NOMEM : TRPDRV_ERR_CUDA, "register: %s",
                          cudaGetErrorString(e));
            } else {
                g_reg[g_nreg].host = c;
                g_reg[g_nreg].bytes = bytes;
                g_reg[g_nreg].dev = dev;
                ++g_nreg;
            }
        }
    }
    pthread_mutex_unlock(&g_di_mu);
    return rc;
}

static int reg_find(const void *ptr)
{
    for (int r = 0; r < g_nreg; ++r)
        if (g_reg[r].host == (const char *)ptr) return r;
    return -1;
}

int trpdrv_refresh_host(const void *ptr)
{
    pthread_mutex_lock(&g_di_mu);
    const int r = reg_find(ptr);
    int rc = TRPDRV_OK;
    if (r < 0) {
        rc = fail(TRPDRV_ERR_ARG, "not a registered array");
    } else {
        cudaSetDevice(g_di.device);
        const cudaError_t e = cudaMemcpy(g_reg[r].dev, g_reg[r].host, g_reg[r].bytes, cudaMemcpyHostToDevice);
        if (e != cudaSuccess) {
            cudaGetLastError();
            rc = fail(TRPDRV_ERR_CUDA, "refresh: %s", cudaGetErrorString(e));
        }
    }
    pthread_mutex_unlock(&g_di_mu);
    return rc;
}

int trpdrv_unregister_host(const void *ptr)
{
    pthread_mutex_lock(&g_di_mu);
    const int r = reg_find(ptr);
    int rc = TRPDRV_OK;
    if (r < 0) {
        rc = fail(TRPDRV_ERR_ARG, "not a registered array");
    } else {
        cudaSetDevice(g_di.device);
        cudaStreamSynchronize(g_di.stream); /* no call in flight reads it */
        cudaFree(g_reg[r].dev);
        g_reg[r] = g_reg[g_nreg - 1];
        memset(&g_reg[g_nreg - 1], 0, sizeof g_reg[0]);
        --g_nreg;
    }
    pthread_mutex_unlock(&g_di_mu);
    return rc;
}

int trpdrv_selftest_bounded_wait(double limit_seconds, int *status, double *elapsed_seconds)
{
    if (!status || !elapsed_seconds) return fail(TRPDRV_ERR_ARG, "selftest: NULL output pointer");
    if (!(limit_seconds > 0.0 && limit_seconds <= 10.0))
        return fail(TRPDRV_ERR_ARG, "selftest: limit %g s outside (0, 10]", limit_seconds);
    int dev = 0;
    TRY(ensure_device(-1, &dev, NULL));
    int *d_status = NULL;
    unsigned long long *d_el = NULL, el = 0;
    int h_status = 0;
    cudaError_t e = cudaMalloc((void **)&d_status, sizeof(int));
    if (e == cudaSuccess) e = cudaMalloc((void **)&d_el, sizeof(unsigned long long));
    if (e == cudaSuccess) e = cudaMemset(d_status, 0, sizeof(int));
    if (e == cudaSuccess)
        e = (cudaError_t)trpdrv_launch_wait_selftest((unsigned long long)(limit_seconds * 1e9), d_status, d_el, NULL);
    if (e == cudaSuccess) e = (cudaError_t)trpdrv_launch_warp_wait_selftest(5000000ull, d_status, NULL);
    if (e == cudaSuccess) e = cudaDeviceSynchronize();
    if (e == cudaSuccess) e = cudaMemcpy(&h_status, d_status, sizeof(int), cudaMemcpyDeviceToHost);
    if (e == cudaSuccess) e = cudaMemcpy(&el, d_el, sizeof el, cudaMemcpyDeviceToHost);
    if (d_status) cudaFree(d_status);
    if (d_el) cudaFree(d_el);
    CUDA_TRY(e);
    *status = h_status;
    *elapsed_seconds = (double)el * 1e-9;
    return TRPDRV_OK;
}

void trpdrv_finalize(void)
{
    pthread_mutex_lock(&g_di_mu);
    di_release();
    pthread_mutex_unlock(&g_di_mu);
    res_close();
}

#define DI_GROW(ptr, cap, count)                                                                    \
    do {                                                                                            \
        if ((size_t)(count) > (cap)) {                                                              \
            if (ptr) cudaFree(ptr);                                                                 \
            ptr = NULL;                                                                             \
            cap = 0;                                                                                \
            CUDA_TRY(cudaMalloc((void **)&(ptr), sizeof(double) * (count)));                        \
            cap = (count);                                                                          \
        }                                                                                           \
    } while (0)

/* Device, stream and the buffers that the energies of one triple of this size need. */
static int di_reserve(int nocc, int nvir, int nbf)
{
    (void)nocc;
    if (!g_di.ready) {
        int dev = 0;
        TRY(ensure_device(-1, &dev, NULL));
        g_di.device = dev;
        CUDA_TRY(cudaStreamCreateWithFlags(&g_di.stream, cudaStreamNonBlocking));
        CUDA_TRY(cudaMalloc((void **)&g_di.tcount, sizeof(unsigned)));
        CUDA_TRY(cudaMemset(g_di.tcount, 0, sizeof(unsigned)));
        CUDA_TRY(cudaMallocHost((void **)&g_di.h_out4, sizeof(double) * 4));
        g_di.ready = 1;
    } else {
        CUDA_TRY(cudaSetDevice(g_di.device));
    }
    DI_GROW(g_di.f, g_di.cap_f, 8 * (size_t)nvir * nvir);
    DI_GROW(g_di.bpart, g_di.cap_part, 4 * (size_t)trpdrv_tengy_pairs(nvir));
    DI_GROW(g_di.vec, g_di.cap_vec, 6 * (size_t)nvir + (size_t)nbf);
    return TRPDRV_OK;
}

static size_t round32(size_t n) { return (n + 31) & ~(size_t)31; }

/* Lays the staging block out for this shape and clears it (the pads must be zero, and mirror and device equal). */
static int di_layout(int ncor, int nocc, int nvir)
{
    if (g_di.cap_stage && g_di.ncor == ncor && g_di.nocc == nocc && g_di.nvir == nvir) return TRPDRV_OK;
    g_di.nvir = 0; /* no valid layout until the end */
    const size_t V = (size_t)nvir, O = (size_t)nocc, ldv = (size_t)row_pitch(nvir), ldo = (size_t)row_pitch(nocc);
    const size_t role[7] = {ldv * V, ldv * V, ldv * V, ldv * O, ldv * O, ldo * V, ldo * V};
    size_t o = 0;
    for (int q = 0; q < DS_N; ++q) {
        g_di.off[q] = o;
        o += round32(q < DS_VEC ? role[q % 7] : q < DS_N - 1 ? V : (size_t)(ncor + nocc + nvir));
    }
    g_di.off[DS_N] = o;
    if (o > g_di.cap_stage) {
        if (g_di.d_stage) cudaFree(g_di.d_stage);
        if (g_di.h_stage) cudaFreeHost(g_di.h_stage);
        g_di.d_stage = g_di.h_stage = NULL;
        g_di.cap_stage = 0;
        CUDA_TRY(cudaMalloc((void **)&g_di.d_stage, sizeof(double) * o));
        CUDA_TRY(cudaMallocHost((void **)&g_di.h_stage, sizeof(double) * o));
        g_di.cap_stage = o;
    }
    CUDA_TRY(cudaStreamSynchronize(g_di.stream)); /* no transfer of a failed call still reads the mirror */
    memset(g_di.h_stage, 0, sizeof(double) * o);
    CUDA_TRY(cudaMemsetAsync(g_di.d_stage, 0, sizeof(double) * o, g_di.stream));
    g_di.ncor = ncor;
    g_di.nocc = nocc;
    g_di.nvir = nvir;
    return TRPDRV_OK;
}

/* Enqueues the transfer of the mirror range [lo, hi) (widened to 16 bytes) to the device block. */
static int di_send(void *ctx, char *lo, char *hi)
{
    (void)ctx;
    const size_t a = ((size_t)(lo - (char *)g_di.h_stage)) & ~(size_t)15;
    const size_t b = ((size_t)(hi - (char *)g_di.h_stage) + 15) & ~(size_t)15;
    CUDA_TRY(cudaMemcpyAsync((char *)g_di.d_stage + a, (char *)g_di.h_stage + a, b - a, cudaMemcpyHostToDevice,
                             g_di.stream));
    return TRPDRV_OK;
}

/* Segments of a call's transfer: the comparison of one runs while the one before crosses the bus. */
#define DI_SEGMENT ((size_t)512 << 10)

/* The energies of the f at g_di.f into g_di.h_out4; waits for them. */
static int di_tengy(int ncor, int nocc, int nvir, double eaijk, const double *const *vec, const double *eorb)
{
    trpdrv_tengy_args ta;
    memset(&ta, 0, sizeof ta);
    ta.ncor = ncor;
    ta.nocc = nocc;
    ta.nvir = nvir;
    ta.use_eaijk = 1;
    ta.eaijk = eaijk;
    ta.f = g_di.f;
    ta.eorb = eorb;
    ta.dintc1 = vec[0];
    ta.dintx1 = vec[1];
    ta.t1v1 = vec[2];
    ta.dintc2 = vec[3];
    ta.dintx2 = vec[4];
    ta.t1v2 = vec[5];
    ta.block_partial = g_di.bpart;
    ta.counter = g_di.tcount;
    ta.out4 = g_di.h_out4;
    LAUNCH_TRY(trpdrv_launch_tengy(&ta, g_di.stream));
    CUDA_TRY(cudaStreamSynchronize(g_di.stream));
    return TRPDRV_OK;
}

/* omp/ccsd_trpdrv_omp_cbody.c:31-145 on the device, for one triple from host buffers. */
static int body_impl(double *f1n, double *f1t, double *f2n, double *f2t, double *f3n, double *f3t, double *f4n,
                     double *f4t, double *eorb, int *ncor_, int *nocc_, int *nvir_, double *emp4_, double *emp5_,
                     int *a_, int *i_, int *j_, int *k_, int *klo_, double *tij, double *tkj, double *tia,
                     double *tka, double *xia, double *xka, double *jia, double *jka, double *kia, double *kka,
                     double *jij, double *jkj, double *kij, double *kkj, double *dintc1, double *dintx1,
                     double *t1v1, double *dintc2, double *dintx2, double *t1v2)
{
    if (!ncor_ || !nocc_ || !nvir_ || !a_ || !i_ || !j_ || !k_ || !klo_ || !emp4_ || !emp5_)
        return fail(TRPDRV_ERR_ARG, "NULL scalar argument");
    const int ncor = *ncor_, nocc = *nocc_, nvir = *nvir_;
    const int a = *a_, i = *i_, j = *j_, k = *k_, klo = *klo_;
    const double *arrays[] = {eorb, tij, tkj, tia, tka, xia, xka, jia, jka, kia, kka,
                              jij, jkj, kij, kkj, dintc1, dintx1, t1v1, dintc2, dintx2, t1v2};
    for (size_t q = 0; q < sizeof arrays / sizeof arrays[0]; ++q)
        if (!arrays[q]) return fail(TRPDRV_ERR_ARG, "NULL array argument #%zu", q);
    if (nocc < 1 || nvir < 1 || ncor < 0 || nocc > TRPDRV_MAX_NOCC || nvir > TRPDRV_MAX_NVIR)
        return fail(TRPDRV_ERR_ARG, "ncor=%d nocc=%d nvir=%d", ncor, nocc, nvir);
    const int nbf = ncor + nocc + nvir;
    if (a < 1 || a > nbf) return fail(TRPDRV_ERR_ARG, "a=%d outside [1,%d]", a, nbf);
    if (i < 1 || i > nocc || j < 1 || j > nocc || k < 1 || k > nocc)
        return fail(TRPDRV_ERR_ARG, "i=%d j=%d k=%d outside [1,%d]", i, j, k, nocc);
    if (klo < 1 || klo > k) return fail(TRPDRV_ERR_ARG, "klo=%d must satisfy 1 <= klo <= k=%d", klo, k);
    const int write_f = env_flag("TRPDRV_WRITE_F", "1");
    if (write_f && (!f1n || !f1t || !f2n || !f2t || !f3n || !f3t || !f4n || !f4t))
        return fail(TRPDRV_ERR_ARG, "TRPDRV_WRITE_F=1 with a NULL f array");

    TRY(di_reserve(nocc, nvir, nbf));
    TRY(di_layout(ncor, nocc, nvir));
    const size_t lnvv = (size_t)nvir * nvir, lnov = (size_t)nocc * nvir, V = (size_t)nvir, O = (size_t)nocc;
    const size_t vv = (size_t)(k - klo) * lnvv, ov = (size_t)(k - klo) * lnov;
    /* the slices in the order of the staging block; slices of registered arrays are read where they are */
    const double *in[DS_N] = {tij, jia, kia, tia, xia, jij, kij, tkj + vv, jka + vv, kka + vv, tka + ov, xka + ov,
                              jkj + ov, kkj + ov, dintc1, dintx1, t1v1, dintc2, dintx2, t1v2, eorb};
    const double *dev[DS_N];
    int ld[DS_N];
    stage_piece pc[DS_N];
    int npi = 0, npk = 0; /* pieces of I from the front, of K and VEC from DS_K on */
    for (int q = 0; q < DS_N; ++q) {
        const int b = q % 7, is_vec = q >= DS_VEC;
        const size_t width = is_vec ? (q < DS_N - 1 ? V : (size_t)nbf) : b < DS_JO ? V : O;
        const size_t rows = is_vec ? 1 : b < DS_TO || b >= DS_JO ? V : O;
        const double *d = reg_lookup(in[q], rows * width);
        ld[q] = (int)width;
        dev[q] = d;
        if (d) continue;
        dev[q] = g_di.d_stage + g_di.off[q];
        const size_t pitch = is_vec ? width : (size_t)row_pitch((int)width);
        ld[q] = (int)pitch;
        stage_piece *p = q < DS_K ? &pc[npi++] : &pc[DS_K + npk++];
        const int flat = pitch == width;
        p->dst = (char *)(g_di.h_stage + g_di.off[q]);
        p->src = (const char *)in[q];
        p->rows = flat ? 1 : rows;
        p->width = sizeof(double) * (flat ? rows * width : width);
        p->pitch = sizeof(double) * (flat ? rows * width : pitch);
    }
    const int threads = stage_threads();
    int rc = stage_send(pc + DS_K, npk, threads, DI_SEGMENT, di_send, NULL);
    if (!rc) rc = stage_send(pc, npi, threads, DI_SEGMENT, di_send, NULL);
    if (rc) {
        g_di.nvir = 0; /* mirror and device may differ now */
        return rc;
    }

    trpdrv_plain_args ga;
    memset(&ga, 0, sizeof ga);
    ga.nocc = nocc;
    ga.nvir = nvir;
    ga.neg2 = 1; /* the reference's alpha = -1 GEMMs */
    ga.f = g_di.f;
    ga.counter = g_di.tcount;
    int vec2 = 1;
    for (int x = 0; x < 8; ++x) { /* f1n f2n f3n f4n f1t f2t f3t f4t: omp/ccsd_trpdrv_omp_cbody.c:70-117 */
        const int A = x < 4 ? DS_I : DS_K, B = x < 4 ? DS_K : DS_I, two = (x >> 1) & 1;
        const int a1 = A + (x & 1 ? DS_KV : DS_J), b1 = B + DS_T, a2 = A + (x & 1 ? DS_XO : DS_TO);
        const int b2 = B + (two ? DS_JO : DS_KO);
        ga.a1[x] = dev[a1];
        ga.b1[x] = dev[b1];
        ga.a2[x] = dev[a2];
        ga.b2[x] = dev[b2];
        ga.lda1[x] = ld[a1];
        ga.ldb1[x] = ld[b1];
        ga.lda2[x] = ld[a2];
        ga.ldb2[x] = ld[b2];
        ga.b1_nt[x] = !two;
        if ((ld[a1] | ld[b1] | ld[a2] | ld[b2]) & 1) vec2 = 0;
        if (((uintptr_t)dev[a1] | (uintptr_t)dev[b1] | (uintptr_t)dev[a2] | (uintptr_t)dev[b2]) & 15u) vec2 = 0;
    }
    LAUNCH_TRY(trpdrv_launch_plain_gemm(&ga, vec2, g_di.stream));

    /* omp/ccsd_trpdrv_omp_cbody.c:122-126 */
    const double eaijk = eorb[a - 1] - (eorb[ncor + i - 1] + eorb[ncor + j - 1] + eorb[ncor + k - 1]);
    TRY(di_tengy(ncor, nocc, nvir, eaijk, dev + DS_VEC, dev[DS_N - 1]));

    if (write_f) {
        double *outs[8] = {f1n, f2n, f3n, f4n, f1t, f2t, f3t, f4t};
        for (int x = 0; x < 8; ++x)
            CUDA_TRY(cudaMemcpy(outs[x], g_di.f + (size_t)x * lnvv, sizeof(double) * lnvv, cudaMemcpyDeviceToHost));
    }
    /* omp/ccsd_trpdrv_omp_cbody.c:133-142 */
    const double e4i = g_di.h_out4[0], e5i = g_di.h_out4[1], e4k = g_di.h_out4[2], e5k = g_di.h_out4[3];
    double emp4 = *emp4_, emp5 = *emp5_;
    emp4 += e4i;
    emp5 += e5i;
    if (i != k) {
        emp4 += e4k;
        emp5 += e5k;
    }
    *emp4_ = emp4;
    *emp5_ = emp5;
    return TRPDRV_OK;
}

static void report(int rc, const char *who)
{
    if (rc == TRPDRV_OK) return;
    if (env_flag("TRPDRV_ON_ERROR", "return")) return;
    fprintf(stderr, "%s: %s: %s\n", who, trpdrv_status_string(rc), t_message);
    abort();
}

#define BODY_ARGS                                                                                   \
    double *f1n, double *f1t, double *f2n, double *f2t, double *f3n, double *f3t, double *f4n, double *f4t, \
        double *eorb, int *ncor, int *nocc, int *nvir, double *emp4, double *emp5, int *a, int *i, int *j,  \
        int *k, int *klo, double *tij, double *tkj, double *tia, double *tka, double *xia, double *xka,     \
        double *jia, double *jka, double *kia, double *kka, double *jij, double *jkj, double *kij,          \
        double *kkj, double *dintc1, double *dintx1, double *t1v1, double *dintc2, double *dintx2,          \
        double *t1v2
#define BODY_PASS                                                                                   \
    f1n, f1t, f2n, f2t, f3n, f3t, f4n, f4t, eorb, ncor, nocc, nvir, emp4, emp5, a, i, j, k, klo, tij, tkj, \
        tia, tka, xia, xka, jia, jka, kia, kka, jij, jkj, kij, kkj, dintc1, dintx1, t1v1, dintc2, dintx2, t1v2

static void body_entry(const char *who, BODY_ARGS)
{
    pthread_mutex_lock(&g_di_mu);
    t_status = TRPDRV_OK;
    const int rc = body_impl(BODY_PASS);
    pthread_mutex_unlock(&g_di_mu);
    report(rc, who);
}

void ccsd_trpdrv_omp_cbody_(BODY_ARGS) { body_entry("ccsd_trpdrv_omp_cbody_", BODY_PASS); }
void ccsd_trpdrv_omp_fbody_(BODY_ARGS) { body_entry("ccsd_trpdrv_omp_fbody_", BODY_PASS); }
void ccsd_trpdrv_cbody_(BODY_ARGS) { body_entry("ccsd_trpdrv_cbody_", BODY_PASS); }
void ccsd_trpdrv_opencl_(BODY_ARGS) { body_entry("ccsd_trpdrv_opencl_", BODY_PASS); }

/* omp/ccsd_tengy_c99.c:5-119 on the device, from host f arrays. */
static int tengy_impl(const double *f1n, const double *f1t, const double *f2n, const double *f2t,
                      const double *f3n, const double *f3t, const double *f4n, const double *f4t,
                      const double *dintc1, const double *dintx1, const double *t1v1, const double *dintc2,
                      const double *dintx2, const double *t1v2, const double *eorb, double eaijk, double *emp4i,
                      double *emp5i, double *emp4k, double *emp5k, int ncor, int nocc, int nvir)
{
    const double *arrays[] = {f1n, f1t, f2n, f2t, f3n, f3t, f4n, f4t, dintc1, dintx1, t1v1, dintc2, dintx2, t1v2, eorb};
    for (size_t q = 0; q < sizeof arrays / sizeof arrays[0]; ++q)
        if (!arrays[q]) return fail(TRPDRV_ERR_ARG, "NULL array argument #%zu", q);
    if (!emp4i || !emp5i || !emp4k || !emp5k) return fail(TRPDRV_ERR_ARG, "NULL output");
    if (nocc < 0 || nvir < 1 || ncor < 0 || nvir > TRPDRV_MAX_NVIR)
        return fail(TRPDRV_ERR_ARG, "ncor=%d nocc=%d nvir=%d", ncor, nocc, nvir);
    const int nbf = ncor + nocc + nvir;
    TRY(di_reserve(nocc > 0 ? nocc : 1, nvir, nbf));
    const size_t lnvv = (size_t)nvir * nvir;
    const double *fs[8] = {f1n, f2n, f3n, f4n, f1t, f2t, f3t, f4t};
    /* the tengy kernel reads the eight f as one contiguous block: always copied */
    for (int x = 0; x < 8; ++x)
        CUDA_TRY(cudaMemcpyAsync(g_di.f + (size_t)x * lnvv, fs[x], sizeof(double) * lnvv, cudaMemcpyHostToDevice,
                                 g_di.stream));
    /* vectors: slices of registered arrays where they are, the others copied */
    const double *vecs[7] = {dintc1, dintx1, t1v1, dintc2, dintx2, t1v2, eorb}, *dvec[7];
    for (int q = 0; q < 7; ++q) {
        const size_t n = q < 6 ? (size_t)nvir : (size_t)nbf;
        dvec[q] = reg_lookup(vecs[q], n);
        if (dvec[q]) continue;
        double *slot = g_di.vec + (size_t)q * nvir;
        CUDA_TRY(cudaMemcpyAsync(slot, vecs[q], sizeof(double) * n, cudaMemcpyHostToDevice, g_di.stream));
        dvec[q] = slot;
    }
    TRY(di_tengy(ncor, nocc, nvir, eaijk, dvec, dvec[6]));
    *emp4i = g_di.h_out4[0];
    *emp5i = g_di.h_out4[1];
    *emp4k = g_di.h_out4[2];
    *emp5k = g_di.h_out4[3];
    return TRPDRV_OK;
}

#define TENGY_ARGS                                                                                  \
    const double *f1n, const double *f1t, const double *f2n, const double *f2t, const double *f3n,       \
        const double *f3t, const double *f4n, const double *f4t, const double *dintc1, const double *dintx1, \
        const double *t1v1, const double *dintc2, const double *dintx2, const double *t1v2,             \
        const double *eorb, const double eaijk, double *emp4i, double *emp5i, double *emp4k, double *emp5k, \
        const int ncor, const int nocc, const int nvir

static void tengy_entry(const char *who, TENGY_ARGS)
{
    pthread_mutex_lock(&g_di_mu);
    t_status = TRPDRV_OK;
    const int rc = tengy_impl(f1n, f1t, f2n, f2t, f3n, f3t, f4n, f4t, dintc1, dintx1, t1v1, dintc2, dintx2, t1v2,
                              eorb, eaijk, emp4i, emp5i, emp4k, emp5k, ncor, nocc, nvir);
    pthread_mutex_unlock(&g_di_mu);
    report(rc, who);
}

void ccsd_tengy_omp(TENGY_ARGS)
{
    tengy_entry("ccsd_tengy_omp", f1n, f1t, f2n, f2t, f3n, f3t, f4n, f4t, dintc1, dintx1, t1v1, dintc2, dintx2,
                t1v2, eorb, eaijk, emp4i, emp5i, emp4k, emp5k, ncor, nocc, nvir);
}

void ccsd_tengy(TENGY_ARGS)
{
    tengy_entry("ccsd_tengy", f1n, f1t, f2n, f2t, f3n, f3t, f4n, f4t, dintc1, dintx1, t1v1, dintc2, dintx2, t1v2,
                eorb, eaijk, emp4i, emp5i, emp4k, emp5k, ncor, nocc, nvir);
}

/* Fortran order (omp/ccsd_tengy_f77.f:1-5): dintc1, dintc2, dintx1, dintx2, t1v1, t1v2, all by reference. */
void ccsd_tengy_omp_(const double *f1n, const double *f1t, const double *f2n, const double *f2t, const double *f3n,
                     const double *f3t, const double *f4n, const double *f4t, const double *dintc1,
                     const double *dintc2, const double *dintx1, const double *dintx2, const double *t1v1,
                     const double *t1v2, const double *eorb, const double *eaijk, double *emp4i, double *emp5i,
                     double *emp4k, double *emp5k, const int *ncor, const int *nocc, const int *nvir)
{
    if (!eaijk || !ncor || !nocc || !nvir) {
        pthread_mutex_lock(&g_di_mu);
        const int rc = fail(TRPDRV_ERR_ARG, "NULL scalar argument");
        pthread_mutex_unlock(&g_di_mu);
        report(rc, "ccsd_tengy_omp_");
        return;
    }
    tengy_entry("ccsd_tengy_omp_", f1n, f1t, f2n, f2t, f3n, f3t, f4n, f4t, dintc1, dintx1, t1v1, dintc2, dintx2,
                t1v2, eorb, *eaijk, emp4i, emp5i, emp4k, emp5k, *ncor, *nocc, *nvir);
}
