/* stage_send of the drop-in staging: the ranges it sends for pieces that follow one another, and for pieces between which
 * a slot is left out.  Returns 0 when every step holds. */
#include <stdio.h>
#include "stage.h"

enum { N = 1 << 20 };
static char mirror[4 * N], device[4 * N], src[N];
static int sends;
static size_t bytes;

static int take(void *ctx, char *lo, char *hi)
{
    (void)ctx;
    ++sends;
    bytes += (size_t)(hi - lo);
    memcpy(device + (lo - mirror), lo, (size_t)(hi - lo));
    return 0;
}

#define CHECK(c)                                                                     \
    do {                                                                             \
        if (!(c)) {                                                                  \
            printf("line %d: %s (%d sends, %zu bytes)\n", __LINE__, #c, sends, bytes); \
            return 1;                                                                \
        }                                                                            \
    } while (0)

static int run(const stage_piece *pc, int n, size_t seg)
{
    sends = 0;
    bytes = 0;
    return stage_send(pc, n, 2, seg, take, NULL);
}

int main(void)
{
    for (int i = 0; i < N; ++i) src[i] = (char)(i * 31 + 7);
    /* a flat piece, padded rows, a flat piece: slots rounded up to 256 bytes, nothing left out */
    stage_piece near[3] = {{mirror, src, 1, 1000, 1000}, {mirror + 1024, src + 1000, 10, 88, 96},
                           {mirror + 2048, src + 2000, 1, 5000, 5000}};
    CHECK(run(near, 3, 1 << 19) == 0 && sends == 1 && bytes == 2048 + 5000);
    CHECK(memcmp(device, mirror, 7048) == 0 && memcmp(device + 2048, src + 2000, 5000) == 0);
    CHECK(run(near, 3, 1 << 19) == 0 && sends == 0); /* nothing changed */
    /* the slot between 4 KB and 2 MB is read elsewhere */
    stage_piece apart[3] = {{mirror, src + 64, 1, 4000, 4000}, {mirror + 2 * N, src, 1, 3000, 3000},
                            {mirror + 2 * N + 3072, src + 3000, 1, 2000, 2000}};
    CHECK(run(apart, 3, 1 << 19) == 0 && sends == 2 && bytes == 4000 + 3072 + 2000);
    CHECK(memcmp(device, src + 64, 4000) == 0 && memcmp(device + 2 * N, src, 3000) == 0 &&
          memcmp(device + 2 * N + 3072, src + 3000, 2000) == 0);
    /* three whole segments and a quarter, then the gap within the last segment */
    const size_t w = (3 << 18) + (1 << 16);
    stage_piece big[2] = {{mirror, src + 1, 1, w, w}, {mirror + 3 * N, src, 1, 100, 100}};
    CHECK(run(big, 2, 1 << 18) == 0 && sends == 5 && bytes == w + 100);
    CHECK(memcmp(device, src + 1, w) == 0 && memcmp(device + 3 * N, src, 100) == 0);
    return 0;
}
