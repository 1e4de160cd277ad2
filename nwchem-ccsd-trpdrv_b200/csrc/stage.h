/*
 * stage.h — host staging of one triple's slices for the drop-in entry points (C and CUDA sources), and the growth of
 * their device buffers.
 *
 * The caller's slices are compared with a pinned mirror and copied where they differ, block by block, so the
 * contents decide what is sent, never a pointer.  Rows may be padded in the mirror (rows of `width` bytes,
 * `pitch` apart).
 */
#ifndef TRPDRV_STAGE_H
#define TRPDRV_STAGE_H

#include <omp.h>
#include <stdlib.h>
#include <string.h>

typedef struct stage_piece {
    char *dst;
    const char *src;
    size_t rows, width, pitch; /* bytes; a contiguous slice is one row */
} stage_piece;

enum { STAGE_BLOCK = 16384 };
/* A single host thread up to this many bytes: it compares and copies them in about the time that waking the team
 * takes.  Above, always the whole team: OpenMP ends and starts threads when the team's size changes. */
enum { STAGE_SERIAL = 256 << 10 };

/* Host threads for the staging copies: TRPDRV_STAGE_THREADS, else up to 16 of OpenMP's. */
static inline int stage_threads(void)
{
    const char *v = getenv("TRPDRV_STAGE_THREADS");
    int n = v ? atoi(v) : 0;
    if (n <= 0) {
        n = omp_get_max_threads();
        if (n > 16) n = 16;
    }
    return n < 1 ? 1 : n;
}

/* Pads and the rounding of slots between two pieces that follow one another, at most. */
enum { STAGE_GAP = 512 };

static inline char *stage_end(const stage_piece *p) { return p->dst + (p->rows - 1) * p->pitch + p->width; }
static inline size_t stage_bytes(const stage_piece *p) { return p->rows * p->width; }

/* Block b of a piece brought up to date; returns 1 if it was written. */
static inline int stage_block(const stage_piece *p, size_t b)
{
    int changed = 0;
    if (p->rows == 1) {
        const size_t lo = b * STAGE_BLOCK, n = p->width - lo < STAGE_BLOCK ? p->width - lo : STAGE_BLOCK;
        if (memcmp(p->dst + lo, p->src + lo, n) != 0) {
            memcpy(p->dst + lo, p->src + lo, n);
            changed = 1;
        }
        return changed;
    }
    const size_t per = p->width < STAGE_BLOCK ? STAGE_BLOCK / p->width : 1;
    const size_t r1 = (b + 1) * per < p->rows ? (b + 1) * per : p->rows;
    for (size_t r = b * per; r < r1; ++r)
        if (memcmp(p->dst + r * p->pitch, p->src + r * p->width, p->width) != 0) {
            memcpy(p->dst + r * p->pitch, p->src + r * p->width, p->width);
            changed = 1;
        }
    return changed;
}

static inline size_t stage_blocks(const stage_piece *p)
{
    if (p->rows == 1) return (p->width + STAGE_BLOCK - 1) / STAGE_BLOCK;
    const size_t per = p->width < STAGE_BLOCK ? STAGE_BLOCK / p->width : 1;
    return (p->rows + per - 1) / per;
}

/* Brings every piece up to date with at most `threads` host threads; returns 1 if anything was written. */
static inline int stage_update(const stage_piece *pc, int npc, int threads)
{
    size_t bytes = 0;
    int nblk = 0, changed = 0;
    for (int q = 0; q < npc; ++q) {
        bytes += stage_bytes(&pc[q]);
        nblk += (int)stage_blocks(&pc[q]);
    }
    if (bytes <= STAGE_SERIAL || threads <= 1) {
        for (int q = 0; q < npc; ++q)
            for (size_t b = 0; b < stage_blocks(&pc[q]); ++b) changed |= stage_block(&pc[q], b);
        return changed;
    }
#pragma omp parallel for num_threads(threads) schedule(static) reduction(| : changed)
    for (int b = 0; b < nblk; ++b) {
        int q = 0;
        size_t r = (size_t)b;
        while (r >= stage_blocks(&pc[q])) r -= stage_blocks(&pc[q++]);
        changed |= stage_block(&pc[q], r);
    }
    return changed;
}

/* Cuts the pieces (ascending dst) into segments of about `seg` bytes and calls send(ctx, lo, hi) for the range
 * [lo, hi) of the mirror that a segment in which something changed covers, as soon as it is up to date: the transfer
 * of one segment runs while the next is compared.  Pieces further apart than the rounding of their slots (what lies
 * between is read elsewhere) go in ranges of their own.  Returns the first non-zero result of send. */
static inline int stage_send(const stage_piece *pc, int npc, int threads, size_t seg,
                             int (*send)(void *ctx, char *lo, char *hi), void *ctx)
{
    enum { MAX_PARTS = 32 };
    stage_piece part[MAX_PARTS];
    int np = 0;
    size_t have = 0;
    for (int q = 0; q < npc; ++q) {
        stage_piece p = pc[q];
        while (p.rows > 0 && p.width > 0) {
            const size_t room = seg > have ? seg - have : 0;
            stage_piece t = p;
            if (p.rows == 1) {
                if (t.width > room && room > 0) t.width = room;
                p.dst += t.width;
                p.src += t.width;
                p.width -= t.width;
            } else {
                size_t n = room / p.width;
                if (n < 1) n = 1;
                if (n < p.rows) t.rows = n;
                p.dst += t.rows * p.pitch;
                p.src += t.rows * p.width;
                p.rows -= t.rows;
            }
            part[np++] = t;
            have += stage_bytes(&t);
            const int done = q == npc - 1 && (p.rows == 0 || p.width == 0);
            if (have >= seg || np == MAX_PARTS || done) {
                if (stage_update(part, np, threads)) {
                    for (int lo = 0, hi = 1; lo < np; lo = hi++) { /* parts lo .. hi - 1 follow one another */
                        while (hi < np && part[hi].dst <= stage_end(&part[hi - 1]) + STAGE_GAP) ++hi;
                        const int e = send(ctx, part[lo].dst, stage_end(&part[hi - 1]));
                        if (e) return e;
                    }
                }
                np = 0;
                have = 0;
            }
        }
    }
    return 0;
}

/* A buffer of at least `want` bytes: kept while its capacity suffices, else released and allocated anew.  A failed
 * allocation leaves neither a buffer nor a capacity, so that the next call, of whatever size, allocates again.
 * Returns the allocator's result. */
static inline int stage_grow(void **p, size_t *cap, size_t want, int (*alloc)(void **p, size_t bytes),
                             void (*release)(void *p))
{
    if (want <= *cap) return 0;
    if (*p) release(*p);
    *p = NULL;
    *cap = 0;
    const int e = alloc(p, want);
    if (e)
        *p = NULL;
    else
        *cap = want;
    return e;
}

#endif /* TRPDRV_STAGE_H */
