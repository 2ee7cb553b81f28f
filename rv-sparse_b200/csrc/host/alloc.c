/*
 * Host allocations of the library, with a failure hook for tests.
 *
 * Every host buffer the library allocates comes from rvsp_malloc /
 * rvsp_calloc / rvsp_realloc.  rvsp_debug_fail_host_alloc(n) (rvsp_debug.h)
 * lets the next n of them succeed and makes the one after return NULL, once,
 * so a test can walk every allocation of a call and check that each failure
 * comes back as RVSP_ERROR_ALLOCATION_FAILED with nothing leaked or half
 * written.  Off (-1) by default: one relaxed atomic load per allocation.
 */
#include <malloc.h>
#include <pthread.h>
#include <stdatomic.h>
#include <stdlib.h>

#include "rvsp_debug.h"
#include "rvsp_internal.h"

static atomic_int g_fail_after = -1;
static atomic_llong g_host_allocs = 0;

/* 1 when this allocation is the one to fail. */
static int inject(void)
{
    atomic_fetch_add_explicit(&g_host_allocs, 1, memory_order_relaxed);
    int cur = atomic_load_explicit(&g_fail_after, memory_order_relaxed);
    while (cur >= 0) {
        if (atomic_compare_exchange_weak(&g_fail_after, &cur, cur - 1))
            return cur == 0;
    }
    return 0;
}

void *rvsp_malloc(size_t n)
{
    return inject() ? NULL : malloc(n);
}

void *rvsp_calloc(size_t n, size_t size)
{
    return inject() ? NULL : calloc(n, size);
}

void *rvsp_realloc(void *p, size_t n)
{
    return inject() ? NULL : realloc(p, n);
}

/*
 * Arrays of one-shot results.  rvsp_csr_destroy keeps the last few large ones
 * here, so that the next product of that size does not fault its pages in
 * again: glibc gives the top of its heap back as soon as it exceeds twice the
 * largest block that was ever mapped, which the three arrays of an FP32 or
 * INT8 result do on every call (1.5 us a page on the measured host: a 19 MB
 * INT8 result 5.4 -> 1.8 ms a call).
 * At most RESULT_KEEP_BYTES in RESULT_KEEP arrays, all plain malloc blocks;
 * the oldest go first.  Arrays are kept only while some thread holds a
 * context of one-shot products (rvsp_result_user): a process that makes none
 * keeps none, and the end of the last such thread gives all of them back, as
 * rvsp_release_kept_results does.
 */
#define RESULT_KEEP 6
#define RESULT_KEEP_BYTES ((size_t)64 << 20)
#define RESULT_MIN_BYTES ((size_t)128 << 10)

static pthread_mutex_t g_kept_lock = PTHREAD_MUTEX_INITIALIZER;
static void *g_kept[RESULT_KEEP]; /* oldest first */
static int g_nkept = 0;
static size_t g_kept_bytes = 0;
static int g_users = 0;

/* Takes entry i out of the list (the lock is held). */
static void *take(int i)
{
    void *p = g_kept[i];
    g_kept_bytes -= malloc_usable_size(p);
    g_nkept--;
    for (; i < g_nkept; i++)
        g_kept[i] = g_kept[i + 1];
    return p;
}

/* rvsp_malloc, out of the kept arrays where one of n to 2 n bytes is there. */
void *rvsp_result_alloc(size_t n)
{
    if (inject())
        return NULL;
    void *p = NULL;
    if (n >= RESULT_MIN_BYTES) {
        int best = -1;
        size_t best_size = 0;
        pthread_mutex_lock(&g_kept_lock);
        for (int i = 0; i < g_nkept; i++) {
            const size_t size = malloc_usable_size(g_kept[i]);
            if (size >= n && size / 2 <= n && (best < 0 || size < best_size)) {
                best = i;
                best_size = size;
            }
        }
        if (best >= 0)
            p = take(best);
        pthread_mutex_unlock(&g_kept_lock);
    }
    return p ? p : malloc(n);
}

/* free(p), or keeps it.  p is any malloc'd block. */
void rvsp_result_free(void *p)
{
    const size_t size = p ? malloc_usable_size(p) : 0;
    if (size < RESULT_MIN_BYTES || size > RESULT_KEEP_BYTES) {
        free(p);
        return;
    }
    void *out[RESULT_KEEP];
    int n = 0;
    pthread_mutex_lock(&g_kept_lock);
    if (g_users > 0) {
        while (g_nkept == RESULT_KEEP || g_kept_bytes + size > RESULT_KEEP_BYTES)
            out[n++] = take(0);
        g_kept[g_nkept++] = p;
        g_kept_bytes += size;
        p = NULL;
    }
    pthread_mutex_unlock(&g_kept_lock);
    free(p);
    while (n > 0)
        free(out[--n]);
}

/* A thread's one-shot context is made (1) or ends (-1). */
void rvsp_result_user(int change)
{
    pthread_mutex_lock(&g_kept_lock);
    g_users += change;
    const int none = g_users == 0;
    pthread_mutex_unlock(&g_kept_lock);
    if (none)
        rvsp_release_kept_results();
}

void rvsp_release_kept_results(void)
{
    void *out[RESULT_KEEP];
    int n = 0;
    pthread_mutex_lock(&g_kept_lock);
    while (g_nkept > 0)
        out[n++] = take(g_nkept - 1);
    pthread_mutex_unlock(&g_kept_lock);
    while (n > 0)
        free(out[--n]);
}

void rvsp_debug_fail_host_alloc(int32_t after)
{
    atomic_store(&g_fail_after, after < 0 ? -1 : (int)after);
}

int64_t rvsp_debug_host_allocs(void)
{
    return (int64_t)atomic_load(&g_host_allocs);
}
