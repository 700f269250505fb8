/* Pageable arrays to and from the device through page-locked pieces.
 *
 * The driver's own way with pageable memory takes 9.4 ms for 100 MB up; in pieces that several threads fill while the one before
 * crosses the link it takes 3.  Page-locking a piece takes 2 to 5 ms, so pieces are kept for the next call: two for the process, given
 * back when its last network goes. */
#include "spg_internal.h"
#include <pthread.h>
#include <string.h>
#define SPG_POOL_PIECES 2

static pthread_mutex_t g_pool_lock = PTHREAD_MUTEX_INITIALIZER;
static void *g_pool[SPG_POOL_PIECES];
static int g_pool_count, g_nets;

static void *piece_take(void)
{
    void *p = NULL;
    pthread_mutex_lock(&g_pool_lock);
    if (g_pool_count) p = g_pool[--g_pool_count];
    pthread_mutex_unlock(&g_pool_lock);
    if (!p && spgk_host_alloc(&p, SPG_STAGE_PIECE) != SPGK_OK) p = NULL;
    return p;
}

static void piece_return(void *p)
{
    if (!p) return;
    pthread_mutex_lock(&g_pool_lock);
    const bool keep = g_nets && g_pool_count < SPG_POOL_PIECES;
    if (keep) g_pool[g_pool_count++] = p;
    pthread_mutex_unlock(&g_pool_lock);
    if (!keep) spgk_host_free(p);
}

/* a network came or went */
void spg_stage_users(int change)
{
    void *drop[SPG_POOL_PIECES];
    int dropped = 0;
    pthread_mutex_lock(&g_pool_lock);
    g_nets += change;
    while (!g_nets && g_pool_count) drop[dropped++] = g_pool[--g_pool_count];
    pthread_mutex_unlock(&g_pool_lock);
    while (dropped) spgk_host_free(drop[--dropped]);
}

/* SPGK_OK or a failed call's code, with nothing held */
int spg_stager_open(spg_stager *s, void *stream)
{
    memset(s, 0, sizeof *s);
    s->stream = stream;
    for (int i = 0; i < 2; i++) {
        s->piece[i] = piece_take();
        const int rc = s->piece[i] ? spgk_event_create(&s->landed[i]) : SPGK_E_NOMEM;
        if (rc) { spg_stager_close(s); return rc; }
    }
    return SPGK_OK;
}

/* waits for the copy from or to a piece */
static int stager_wait(spg_stager *s, int i)
{
    if (!s->busy[i]) return SPGK_OK;
    s->busy[i] = false;
    const int rc = spgk_event_sync(s->landed[i]);
    if (rc) s->unsure = true;
    return rc;
}

/* a copy from or to a piece has been queued */
static int stager_queued(spg_stager *s, int i)
{
    const int rc = spgk_event_record(s->landed[i], s->stream);
    if (rc) s->unsure = true;
    else s->busy[i] = true;
    return rc;
}

/* the piece whose turn it is, once the device has done with what it held */
static int stager_turn(spg_stager *s, int *turn)
{
    const int i = *turn = s->turn;
    s->turn ^= 1;
    return stager_wait(s, i);
}

void spg_stager_close(spg_stager *s)
{
    for (int i = 0; i < 2; i++) stager_wait(s, i);
    const bool idle = !s->unsure || spgk_stream_sync(s->stream) == SPGK_OK;
    for (int i = 0; i < 2; i++) {
        if (s->landed[i]) spgk_event_destroy(s->landed[i]);
        if (idle) piece_return(s->piece[i]);
        else spgk_host_free(s->piece[i]);
        s->landed[i] = s->piece[i] = NULL;
    }
}

/* host memory to the device: `src` may be changed as soon as this returns */
int spg_stager_up(spg_stager *s, void *dev, const void *src, size_t bytes)
{
    for (size_t at = 0; at < bytes; at += SPG_STAGE_PIECE) {
        const size_t n = bytes - at < SPG_STAGE_PIECE ? bytes - at : SPG_STAGE_PIECE;
        int i, rc = stager_turn(s, &i);
        if (rc) return rc;
        spg_stage_copy(s->piece[i], (const char *)src + at, n);
        if ((rc = spgk_memcpy_h2d((char *)dev + at, s->piece[i], n, s->stream)) || (rc = stager_queued(s, i))) return rc;
    }
    return SPGK_OK;
}

/* device memory to `sink`, segment by segment and piece by piece in order; complete when this returns.  A sink that fails ends it with
 * SPGK_E_ARG. */
int spg_stager_down(spg_stager *s, spg_sink_fn sink, const spg_segment *seg, int count)
{
    struct { int piece, seg; size_t at, n; } now, before = { -1, 0, 0, 0 };
    int g = 0;
    size_t at = 0;
    for (;;) {
        int rc;
        while (g < count && at >= seg[g].bytes) { g++; at = 0; }
        now.piece = -1;
        if (g < count) {
            now.seg = g; now.at = at; now.n = seg[g].bytes - at < SPG_STAGE_PIECE ? seg[g].bytes - at : SPG_STAGE_PIECE;
            at += now.n;
            if ((rc = stager_turn(s, &now.piece)) || (rc = spgk_memcpy_d2h(s->piece[now.piece], (const char *)seg[g].dev + now.at, now.n, s->stream)) ||
                (rc = stager_queued(s, now.piece))) return rc;
        }
        if (before.piece >= 0) {
            if ((rc = stager_wait(s, before.piece))) return rc;
            if (!sink(seg[before.seg].ctx, before.at, s->piece[before.piece], before.n)) return SPGK_E_ARG;
        }
        if (now.piece < 0) return SPGK_OK;
        before.piece = now.piece; before.seg = now.seg; before.at = now.at; before.n = now.n;
    }
}

/* a sink that fills the array `ctx` */
bool spg_sink_array(void *ctx, size_t at, const void *piece, size_t n)
{
    spg_bulk_copy((char *)ctx + at, piece, n);
    return true;
}
