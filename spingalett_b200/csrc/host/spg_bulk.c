/* Bulk host work on several threads: copies into page-locked staging, reading and decoding files.
 *
 * One thread copies 11 to 16 GB/s and takes a page fault for every 4 KB of fresh memory it writes; the host link takes
 * 52 GB/s.  Measured on 16 cores, 188 MB from pageable memory into two page-locked buffers: 5.4 ms with eight threads and
 * memcpy, 3.7 with stores that do not read the destination first, 2.8 with twelve threads. */
#include "spg_internal.h"
#include <pthread.h>
#include <stdatomic.h>
#include <stdlib.h>
#include <string.h>
#include <sys/mman.h>
#include <unistd.h>
#if defined(__x86_64__)
#include <immintrin.h>
#endif

#define SPG_BULK_THREADS 16    /* most for a caller; SPINGALETT_STAGE_THREADS in the environment asks for another number of them */

static atomic_int g_callers;   /* calls with several threads that are at work in the process */

typedef struct { spg_slice_fn fn; void *ctx; size_t lo, hi; } slice;

static void *slice_worker(void *arg)
{
    slice *s = arg;
    s->fn(s->ctx, s->lo, s->hi);
    return NULL;
}

/* The cores are shared by all callers: a batch cut over several devices has one for each of them. */
static int bulk_threads(int callers)
{
    const char *e = getenv("SPINGALETT_STAGE_THREADS");
    const long cores = sysconf(_SC_NPROCESSORS_ONLN);
    int want = e && atoi(e) > 0 ? atoi(e) : (int)(cores - cores / 4) / callers;      /* three quarters: the caller's program lives here too */
    if (want < 1) want = 1;
    return want > SPG_BULK_THREADS ? SPG_BULK_THREADS : want;
}

static void run_slices(spg_slice_fn fn, void *ctx, size_t n, size_t grain, size_t nt)
{
    const size_t share = ((n + nt - 1) / nt + grain - 1) / grain * grain;
    pthread_t th[SPG_BULK_THREADS];
    slice sl[SPG_BULK_THREADS];
    size_t started = 0;
    for (size_t t = 1; t < nt && t * share < n; t++) {
        const size_t lo = t * share;
        sl[t] = (slice){ fn, ctx, lo, n - lo < share ? n : lo + share };
        if (pthread_create(&th[t], NULL, slice_worker, &sl[t]) != 0) { fn(ctx, lo, n); break; }      /* no thread: this one does the rest */
        started = t;
    }
    fn(ctx, 0, share < n ? share : n);
    for (size_t t = 1; t <= started; t++) pthread_join(th[t], NULL);
}

/* fn over [0, n) in slices that start at multiples of `grain`; a thread for every `least` of n at most */
void spg_bulk(spg_slice_fn fn, void *ctx, size_t n, size_t grain, size_t least)
{
    size_t nt = n / least;
    if (nt < 2) { fn(ctx, 0, n); return; }
    const size_t most = (size_t)bulk_threads(atomic_fetch_add(&g_callers, 1) + 1);
    if (nt > most) nt = most;
    if (nt < 2) fn(ctx, 0, n);
    else run_slices(fn, ctx, n, grain, nt);
    atomic_fetch_sub(&g_callers, 1);
}

#if defined(__x86_64__)
/* dst on a 32-byte boundary: stores that leave the destination's lines out of the caches, where nobody will look for them */
__attribute__((target("avx2"))) static void copy_streaming(char *dst, const char *src, size_t n)
{
    size_t i = 0;
    for (; i + 128 <= n; i += 128) {
        const __m256i a = _mm256_loadu_si256((const __m256i *)(src + i)), b = _mm256_loadu_si256((const __m256i *)(src + i + 32));
        const __m256i c = _mm256_loadu_si256((const __m256i *)(src + i + 64)), d = _mm256_loadu_si256((const __m256i *)(src + i + 96));
        _mm256_stream_si256((__m256i *)(dst + i), a);
        _mm256_stream_si256((__m256i *)(dst + i + 32), b);
        _mm256_stream_si256((__m256i *)(dst + i + 64), c);
        _mm256_stream_si256((__m256i *)(dst + i + 96), d);
    }
    _mm_sfence();
    memcpy(dst + i, src + i, n - i);
}
#endif

typedef struct { char *dst; const char *src; } copy_ctx;
static void copy_slice(void *ctx, size_t lo, size_t hi)
{
    const copy_ctx *c = ctx;
#if defined(__x86_64__)
    if (((uintptr_t)(c->dst + lo) & 31u) == 0 && __builtin_cpu_supports("avx2")) { copy_streaming(c->dst + lo, c->src + lo, hi - lo); return; }
#endif
    memcpy(c->dst + lo, c->src + lo, hi - lo);
}

/* into page-locked memory that the device reads next */
void spg_stage_copy(void *dst, const void *src, size_t bytes)
{
    copy_ctx c = { dst, src };
    if (bytes < SPG_STAGE_THREADED) memcpy(dst, src, bytes);
    else spg_bulk(copy_slice, &c, bytes, 4096, (size_t)1 << 20);
}

/* Long fresh memory in pages of 2 MB where the system has them: it is filled once, and a page fault for every 4 KB of 100 MB takes as long
 * as filling it. */
void spg_large_pages(void *p, size_t bytes)
{
    const uintptr_t page = (uintptr_t)2 << 20, lo = ((uintptr_t)p + page - 1) & ~(page - 1), hi = ((uintptr_t)p + bytes) & ~(page - 1);
    if (p && hi > lo) madvise((void *)lo, hi - lo, MADV_HUGEPAGE);
}

/* into memory that the host reads next */
static void plain_slice(void *ctx, size_t lo, size_t hi)
{
    const copy_ctx *c = ctx;
    memcpy(c->dst + lo, c->src + lo, hi - lo);
}

void spg_bulk_copy(void *dst, const void *src, size_t bytes)
{
    copy_ctx c = { dst, src };
    spg_bulk(plain_slice, &c, bytes, 4096, (size_t)1 << 20);
}

static void zero_slice(void *ctx, size_t lo, size_t hi) { memset((char *)ctx + lo, 0, hi - lo); }
void spg_bulk_zero(void *dst, size_t bytes) { spg_bulk(zero_slice, dst, bytes, 4096, (size_t)1 << 20); }
