/*
 * Internal interface between the C host layer (host.c) and the CUDA translation units.
 * Plain C structs and extern "C" launchers only; every launcher enqueues on the given stream and
 * returns a cudaError_t value (0 = success).
 */
#ifndef TRPDRV_LAUNCH_H
#define TRPDRV_LAUNCH_H

#include <stddef.h>
#include <stdint.h>

#ifdef __cplusplus
extern "C" {
#endif

/* Width of the (b,c) tiles of the fused kernel. */
#define TRPDRV_TILE 32
/* Energy slots per fused work item (one per warp of the fused CTA). */
#define TRPDRV_FUSED_SLOTS 8
/* Triples are packed as (i-1) | (j-1) << 10 | (k-1) << 20 (0-based), so nocc must be < 1024. */
#define TRPDRV_MAX_NOCC 1023
/* Largest nvir the kernels accept (index arithmetic is 32-bit within one nvir x nvir block). */
#define TRPDRV_MAX_NVIR 16384

/* Device view of one system in a plan.  ntov/nxov hold -tov/-xov, so that every f is the sum of
 * two products accumulated with +1 (the reference's alpha = -1 GEMMs, omp/ccsd_trpdrv_omp_cbody.c:73-116). */
typedef struct trpdrv_dev_system {
    int ncor, nocc, nvir, a;
    int nb;              /* ceil(nvir / TRPDRV_TILE) */
    int npairs;          /* nb*(nb+1)/2 tile pairs (B <= C) */
    int64_t ntriples;    /* records of this system in the plan: n_a * nt */
    int64_t nt;          /* triples per a (this rank's share): the length of `triples` and `order` */
    int n_a;             /* virtual indices a .. a + n_a - 1 swept (1 = the reference driver's single a) */
    int ldv, ldo;        /* cp.async staging: leading dimension of the rows of nvir (t2, jvv, kvv, ntov, nxov) and of
                            nocc (jov, kov) doubles; 0 = nvir / nocc (packed, as callers hold them).  The
                            plans pad odd rows to the next even length (trpdrv_launch_pack_rows). */
    int pack_edge;       /* 1: the last tile holds 1..16 valid virtual indices and the TMA kernel runs the
                            edge pairs (B, E), (B + 1, E) (B even) as one packed work item; the item of
                            (B + 1, E) is then skipped (its energy slots are written by the packed one) */
    int64_t item_begin;  /* first fused work item of this system */
    const double *eorb, *t2, *jvv, *kvv, *ntov, *nxov, *jov, *kov, *dintc, *dintx, *t1v;
    const int32_t *triples; /* packed triples, driver order (energies are stored in this order) */
    const int32_t *order;   /* fused kernels: processing position -> triple index, or NULL (identity) */
    double *partial;        /* [ntriples*npairs][TRPDRV_FUSED_SLOTS][4]: e4i, e5i, e4k, e5k */
    double *rec;            /* [ntriples][4] per triple */
} trpdrv_dev_system;

/* Fused persistent kernel (fused_tma.cu): grid CTAs (one per SM) pull (triple, tile pair) items from
 * *counter (must be 0 at launch) and write per-item energies.  *status bit 0: malformed queue entry; bit 1: a
 * pipeline wait ran out.  pair_major = 1: a system's items run pair by pair over all its triples instead of triple
 * by triple (whole systems only: item ranges no longer follow the processing order).  Two stagings of the operands feed the same MMA loop:
 *   trpdrv_launch_fused: cp.async; any sizes, any number of systems.  vec2 = 1 (16-byte copies) requires
 *     even nvir and nocc and 16-byte aligned tensors for every system; mma_k selects the FP64 MMA shape
 *     m16n8k4 (4) or m16n8k8 (8).
 *   trpdrv_launch_fused_tma: TMA; even nvir and nocc, 16-byte aligned tensors and at most
 *     TRPDRV_TMA_MAX_SYSTEMS systems (trpdrv_tma_supported); mma_k 8 or 16.  trpdrv_tma_prepare encodes the
 *     tensor maps of every system into a host blob of trpdrv_tma_maps_bytes() bytes (64-byte aligned)
 *     that each launch passes by value. */
int trpdrv_launch_fused(const trpdrv_dev_system *d_sys, int nsys, int64_t total_items, int pair_major,
                        unsigned long long *counter, int *status, int grid, int vec2, int mma_k,
                        void *stream);
#define TRPDRV_TMA_MAX_SYSTEMS 8
int trpdrv_tma_supported(const trpdrv_dev_system *h_sys, int nsys);
/* 1 if the fused kernel packs the edge pairs of a system with this nvir (see pack_edge). */
int trpdrv_tma_pack_edge(int nvir);
size_t trpdrv_tma_maps_bytes(void);
int trpdrv_tma_prepare(const trpdrv_dev_system *h_sys, int nsys, void *maps_out);
int trpdrv_launch_fused_tma(const trpdrv_dev_system *d_sys, int nsys, int64_t total_items, int pair_major,
                            unsigned long long *counter, int *status, int grid, const void *maps,
                            int mma_k, void *stream);
int trpdrv_fused_tma_init(void);
/* One thread waits, with the production bounded wait and the given limit, on an mbarrier that
 * nothing completes: sets bit 1 of *status when the wait gives up (bit 2 if it wrongly completes)
 * and stores how long it waited. */
int trpdrv_launch_wait_selftest(unsigned long long limit_ns, int *status, unsigned long long *elapsed_ns,
                                void *stream);

/* One warp waits as the emulated form's warps do, half of its lanes with a shorter limit than the phase takes: bit 3 of
 * *status unless all lanes give up together. */
int trpdrv_launch_warp_wait_selftest(unsigned long long limit_ns, int *status, void *stream);

/* Emulated-FP64 (Ozaki int8) form, ozaki.cu.  Per system: digit slices of the A operands
 * sa [nocc][slices][2 nvir][dp] and of the B operands sb [nocc*nocc][slices][2 nvir][dp] (int8,
 * dp = trpdrv_oz_dp: nvir + nocc rounded up to 32), with power-of-two scales ea [nocc][2 nvir] and
 * eb [nocc*nocc][2 nvir].  trpdrv_oz_prepare encodes the two tensor maps into a host blob of
 * trpdrv_oz_maps_bytes() bytes (64-byte aligned).  A batch is npos consecutive positions of the
 * system's processing order starting at pos0: the contraction kernel writes their f into
 * fbuf [npos][8][nvir][trpdrv_oz_ldf(nvir)] and the tengy kernel writes the sums of each 16-wide tile pair into
 * one slot of the triple's items in `partial` (the other slots must be zero), for
 * trpdrv_launch_records.  *status as the fused kernels (bit 0 malformed entry, bit 1 a wait
 * ran out).  The contraction kernel is persistent: grid = CTAs (one per SM). */
#define TRPDRV_OZ_MIN_SLICES 4
#define TRPDRV_OZ_MAX_SLICES 8
typedef struct trpdrv_oz_system {
    int nocc, nvir, slices, dp, n_a;  /* n_a: a values swept; sa holds n_a * nocc planes */
    signed char *sa, *sb;
    double *ea, *eb;
    int32_t *jobs;  /* the products of every position in order, position << 1 | group: group 0 (n: SA[i] SB[j,k])
                       and, unless i == k, group 1 (t: SA[k] SB[j,i]); with i == k group 0 stores both */
} trpdrv_oz_system;
/* Doubles between the columns of f in a batch buffer: nvir rounded up to even (16-byte rows for TMA). */
#ifdef __CUDACC__
__host__ __device__
#endif
static inline int trpdrv_oz_ldf(int nvir) { return nvir + (nvir & 1); }
int trpdrv_oz_slices_supported(int slices);
int trpdrv_oz_dp(int nocc, int nvir);
size_t trpdrv_oz_maps_bytes(void);
int trpdrv_oz_prepare(const trpdrv_oz_system *oz, void *maps_out);
int trpdrv_launch_oz_slices(const trpdrv_dev_system *h_sys, const trpdrv_oz_system *oz, void *stream);
/* Products oz->jobs[job0 .. job0 + njobs) (those of consecutive positions from pos0) into fbuf; enpos > 0 (requires
 * trpdrv_oz_fused_energy_supported(nvir)): the same launch's energy warps also compute the energies
 * of positions epos0 .. epos0 + enpos - 1, whose f an earlier launch stored at efbuf.  njobs = 0 gives an
 * energies-only launch. */
int trpdrv_launch_oz_gemm(const trpdrv_dev_system *h_sys, const trpdrv_oz_system *oz, const void *maps,
                          int64_t pos0, int64_t job0, int njobs, double *fbuf, int64_t epos0, int enpos,
                          const double *efbuf, int *status, int grid, void *stream);
int trpdrv_oz_fused_energy_supported(int nvir);
/* The energies as a launch of their own (odd nvir, or TRPDRV_OZ_FUSED_ENERGY=0).
 * The plans launch the energies of one batch on a second stream, ordered only after that batch's products.  The
 * tiles arrive by TMA (fbuf 16-byte aligned), with a bounded wait that sets *status bit 1 when it runs out;
 * with TRPDRV_OZ_TENGY_TMA=0 by cp.async. */
int trpdrv_launch_oz_tengy(const trpdrv_dev_system *h_sys, int64_t pos0, int npos, const double *fbuf, int *status,
                           void *stream);
int trpdrv_oz_init(void);

/* Per-triple sums of the per-item energies of nsys systems (descriptors on host and device): partial -> rec. */
int trpdrv_launch_records(const trpdrv_dev_system *h_sys, const trpdrv_dev_system *d_sys, int nsys, void *stream);

/* Each system's compensated total over rec, of emp4i + [i != k] emp4k summed over the triples:
 * res[4 s ..] = emp4 hi, emp4 lo, emp5 hi, emp5 lo; res[4 nsys] = the value of *status.  res is pinned host memory
 * (device-accessible).  bsum: trpdrv_totals_doubles doubles; done: nsys zeros (left at zero).  Systems
 * without records are not written. */
size_t trpdrv_totals_doubles(const trpdrv_dev_system *h_sys, int nsys);
int trpdrv_launch_totals(const trpdrv_dev_system *h_sys, const trpdrv_dev_system *d_sys, int nsys, double *bsum,
                         unsigned *done, const int *status, double *res, void *stream);

/* dst[i] = -src[i]. */
int trpdrv_launch_negate(const double *src, double *dst, size_t n, void *stream);

/* Rows copied to an even pitch: dst[r * pitch + c] = src[r * width + c] (negated where neg), zeros for
 * c >= width, for every segment s < n and r < rows, in one launch.  pitch even, dst 16-byte aligned. */
#define TRPDRV_PACK_LIST_MAX 8
typedef struct trpdrv_pack_list {
    int n;
    struct {
        const double *src;
        double *dst;
        long long rows;
        int width, pitch, neg;
    } seg[TRPDRV_PACK_LIST_MAX];
} trpdrv_pack_list;
int trpdrv_launch_pack_rows(const trpdrv_pack_list *list, void *stream);

/* Plain path.  Single triple: one grouped launch computes the eight f = A1*op(B1) + A2*B2 (neg2: - A2*B2) into
 * f[8][nvir][nvir] (order f1n f2n f3n f4n f1t f2t f3t f4t); b1_nt[x] = 1 if B1 is used transposed.  counter, if
 * not NULL, is zeroed for the trpdrv_launch_tengy that follows on the stream. */
typedef struct trpdrv_plain_args {
    int nocc, nvir, neg2;
    const double *a1[8], *b1[8], *a2[8], *b2[8];
    int lda1[8], ldb1[8], lda2[8], ldb2[8]; /* even for vec2 */
    int b1_nt[8];
    double *f;
    unsigned *counter;
} trpdrv_plain_args;
int trpdrv_launch_plain_gemm(const trpdrv_plain_args *args, int vec2, void *stream);

/* Tile pairs trpdrv_launch_tengy sums one by one (the length of block_partial in fours). */
int64_t trpdrv_tengy_pairs(int nvir);
/* Standalone tengy over f[8][nvir][nvir] on the device.  eaijk is taken from `eaijk` when
 * use_eaijk != 0, else computed on the device from eorb and the 1-based a, i, j, k.  Writes
 * out4[0..3] = emp4i, emp5i, emp4k, emp5k.  block_partial needs 4*trpdrv_tengy_pairs(nvir) doubles, counter
 * one zeroed unsigned int (it is left at zero again).  Launched as a programmatic dependent of the launch
 * before it on the stream, which must be what writes f (or no kernel). */
typedef struct trpdrv_tengy_args {
    int ncor, nocc, nvir;
    int use_eaijk;
    double eaijk;
    int a, i, j, k;
    const double *f;
    const double *eorb, *dintc1, *dintx1, *t1v1, *dintc2, *dintx2, *t1v2;
    double *block_partial;
    unsigned int *counter;
    double *out4;
} trpdrv_tengy_args;
int trpdrv_launch_tengy(const trpdrv_tengy_args *args, void *stream);

/* Records pos0 .. pos0 + n - 1 of a plan's system: f into f[n][8][nvir][nvir], then the energies into
 * h_sys->rec.  block_partial: n * 4 * trpdrv_tengy_pairs(nvir) doubles; counter: n zeros (left at zero).
 * trpdrv_plain_batch: the batch plans use for this nvir.  vec2 as for the fused kernel.  chained: the launch
 * before it on the stream is the same system's previous batch, whose energies this one's products may overlap. */
int trpdrv_plain_batch(int nvir);
int trpdrv_launch_plain_batch(const trpdrv_dev_system *h_sys, int64_t pos0, int n, double *f, double *block_partial,
                              unsigned *counter, int vec2, int chained, void *stream);

/* Sets the dynamic shared memory limits of every kernel (call once per device). */
int trpdrv_kernels_init(void);

/* Sets the calling thread's trpdrv_last_error() status and message; returns status. */
int trpdrv_record_error(int status, const char *message);

#ifdef __cplusplus
}
#endif
#endif
