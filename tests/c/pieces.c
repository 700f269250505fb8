/* A page-locked piece is handed to the next user only once the copies from and to it are known to be over, also where an event could not be recorded
 * behind one or a call failed half way; otherwise it is given back to the driver, which waits for them.  Host code of the library on fake
 * kernels, as in unread_status.c; a copy is under way until its stream or an event behind it has been waited for. */
#include <stdio.h>
#include <stdlib.h>
#include <string.h>
#include "spg_internal.h"

static int g_calls, g_fail_at;                 /* the call that fails, of those that may */
static const void *g_under_way[64];
static int g_count;
static bool fails(void) { return ++g_calls == g_fail_at; }

int spgk_host_alloc(void **p, size_t bytes) { *p = malloc(bytes); return 0; }
static void over(const void *p) { for (int i = 0; i < g_count; i++) if (g_under_way[i] == p) g_under_way[i--] = g_under_way[--g_count]; }
int spgk_host_free(void *p) { over(p); free(p); return 0; }
int spgk_event_create(void **e) { *e = calloc(1, sizeof(int)); return 0; }
int spgk_event_destroy(void *e) { free(e); return 0; }
int spgk_event_record(void *e, void *s) { (void)s; if (fails()) return SPGK_E_CUDA; *(int *)e = g_count; return 0; }
/* (an event that was never recorded behind the copy says nothing about it) */
int spgk_event_sync(void *e) { if (fails()) return SPGK_E_CUDA; if (*(int *)e >= g_count) g_count = 0; *(int *)e = 0; return 0; }
int spgk_stream_sync(void *s) { (void)s; if (fails()) return SPGK_E_CUDA; g_count = 0; return 0; }
int spgk_memcpy_h2d(void *d, const void *h, size_t bytes, void *s) { (void)d; (void)bytes; (void)s; if (fails()) return SPGK_E_CUDA; g_under_way[g_count++] = h; return 0; }
int spgk_memcpy_d2h(void *h, const void *d, size_t bytes, void *s) { (void)d; (void)bytes; (void)s; if (fails()) return SPGK_E_CUDA; g_under_way[g_count++] = h; return 0; }

static bool sink(void *ctx, size_t at, const void *piece, size_t n) { (void)ctx; (void)at; (void)piece; (void)n; return !fails(); }

int main(void)
{
    static char data[3 * SPG_STAGE_PIECE + 5];
    spg_stage_users(1);
    for (int down = 0; down < 2; down++)
        for (g_fail_at = 1; g_fail_at < 24; g_fail_at++) {
            spg_stager s;
            g_calls = 0;
            if (spg_stager_open(&s, NULL)) return 2;
            const spg_segment seg = { data, sizeof data, NULL };
            const int rc = down ? spg_stager_down(&s, sink, &seg, 1) : spg_stager_up(&s, data, data, sizeof data);
            spg_stager_close(&s);
            const int failed = g_calls >= g_fail_at;
            if (!failed && rc) return 3;
            /* what the next user gets is not under way */
            if (spg_stager_open(&s, NULL)) return 4;
            for (int i = 0; i < 2; i++)
                for (int k = 0; k < g_count; k++)
                    if (g_under_way[k] == s.piece[i]) { printf("%s, call %d failed: a piece in use is handed out\n", down ? "down" : "up", g_fail_at); return 1; }
            g_count = 0;
            spg_stager_close(&s);
        }
    spg_stage_users(-1);
    puts("every piece at rest");
    return 0;
}
