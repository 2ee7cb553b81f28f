/*
 * numpy arrays that take over the memory of a one-shot result (rvsp/api.py).
 *
 * An array owns its memory, and can be resized in place, when numpy allocated
 * it, by the allocator that is set at the time (PyDataMem_Handler, NEP 49),
 * which numpy keeps for the array's resize and free.  So the array is made
 * while this allocator is set, whose malloc hands out the result's block;
 * free goes where rvsp_csr_destroy's does.  A copy instead took 0.4 ms for
 * 5 MB and, in fresh pages, 4 ms for 19 MB.
 *
 * numpy's C API is called through the table in its capsule (the library is
 * built without Python's and numpy's headers).
 */
#include <stdlib.h>

#include "rvsp_internal.h"

/* places in numpy's table, which keep their meaning */
enum { DESCR_FROM_TYPE = 45, EMPTY = 184 };

static _Thread_local void *g_block; /* handed out by the next malloc */

static void *block_malloc(void *ctx, size_t n)
{
    (void)ctx;
    void *p = g_block;
    g_block = NULL;
    return p ? p : malloc(n);
}

static void *block_calloc(void *ctx, size_t n, size_t size)
{
    (void)ctx;
    return calloc(n, size);
}

static void *block_realloc(void *ctx, void *p, size_t n)
{
    (void)ctx;
    return realloc(p, n);
}

static void block_free(void *ctx, void *p, size_t n)
{
    (void)ctx;
    (void)n;
    rvsp_result_free(p);
}

/* numpy's PyDataMem_Handler, version 1 */
static struct {
    char name[127];
    uint8_t version;
    void *ctx;
    void *(*malloc)(void *, size_t);
    void *(*calloc)(void *, size_t, size_t);
    void *(*realloc)(void *, void *, size_t);
    void (*free)(void *, void *, size_t);
} g_handler = {"rvsp_result", 1, NULL, block_malloc, block_calloc, block_realloc, block_free};

void *rvsp_numpy_handler(void)
{
    return &g_handler;
}

/* A one-dimensional array of n > 0 elements of numpy's type number over the
 * malloc block p.  The caller holds the GIL and has set the handler; no Python
 * code runs between here and the allocation. */
void *rvsp_numpy_array(void *const *api, int type, intptr_t n, void *p)
{
    void *(*descr_from_type)(int) = (void *(*)(int))api[DESCR_FROM_TYPE];
    void *(*empty)(int, const intptr_t *, void *, int) =
        (void *(*)(int, const intptr_t *, void *, int))api[EMPTY];
    void *descr = descr_from_type(type);
    g_block = p;
    void *array = empty(1, &n, descr, 0);
    g_block = NULL;
    return array;
}
