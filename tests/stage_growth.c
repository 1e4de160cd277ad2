/* stage_grow of the drop-in staging with an allocator that fails on request: what is left after a failure, and what
 * the next, smaller call does.  Prints nothing and returns 0 when every step holds. */
#include <stdio.h>
#include "stage.h"

static int fails, allocs, live;

static int stub_alloc(void **p, size_t bytes)
{
    if (fails > 0) {
        --fails;
        *p = (void *)16; /* whatever a failing allocator leaves there is not used */
        return 2;
    }
    ++allocs;
    ++live;
    *p = malloc(bytes);
    return *p ? 0 : 2;
}

static void stub_release(void *p)
{
    --live;
    free(p);
}

#define CHECK(c)                                             \
    do {                                                     \
        if (!(c)) {                                          \
            printf("line %d: %s\n", __LINE__, #c);           \
            return 1;                                        \
        }                                                    \
    } while (0)

int main(void)
{
    void *p = NULL;
    size_t cap = 0;
    CHECK(stage_grow(&p, &cap, 100, stub_alloc, stub_release) == 0 && p && cap == 100 && allocs == 1);
    void *first = p;
    CHECK(stage_grow(&p, &cap, 60, stub_alloc, stub_release) == 0 && p == first && allocs == 1);
    fails = 1;
    CHECK(stage_grow(&p, &cap, 200, stub_alloc, stub_release) == 2);
    CHECK(p == NULL && cap == 0 && live == 0);
    CHECK(stage_grow(&p, &cap, 60, stub_alloc, stub_release) == 0); /* smaller than the lost buffer */
    CHECK(p != NULL && cap == 60 && allocs == 2 && live == 1);
    memset(p, 1, 60);
    CHECK(stage_grow(&p, &cap, 100, stub_alloc, stub_release) == 0 && p && cap == 100 && live == 1);
    stub_release(p);
    return 0;
}
