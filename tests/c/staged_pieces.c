/* Staged host batches with short last chunks: every row arrives, in copies that get somewhere, and a chunk is only cut where
 * its pieces are long enough to be staged by several threads (4 MB).  Host code of the library on fake
 * kernels, as in unread_status.c; "device memory" is the heap, and the fake copy looks at what it is given. */
#include <stdio.h>
#include <stdlib.h>
#include <string.h>
#include "spingalett_b200.h"
#include "spingalett_b200_kernels.h"

#define CHUNK ((size_t)16384)
static const float *g_in;                      /* the call's inputs while one is being watched, their size and row */
static size_t g_rows, g_row_bytes, g_at, g_copies;

int spgk_device_count(int *n) { *n = 1; return 0; }
int spgk_get_device(int *d) { *d = 0; return 0; }
int spgk_malloc(void **p, size_t bytes) { *p = malloc(bytes); return 0; }
int spgk_free(void *p) { free(p); return 0; }
int spgk_host_alloc(void **p, size_t bytes) { *p = aligned_alloc(64, (bytes + 63) & ~(size_t)63); return 0; }
int spgk_host_free(void *p) { free(p); return 0; }
int spgk_memset(void *p, int v, size_t bytes, void *s) { (void)s; memset(p, v, bytes); return 0; }
int spgk_is_device_pointer(const void *p) { (void)p; return 0; }
int spgk_is_pinned_host_pointer(const void *p) { (void)p; return 0; }
const char *spgk_error_string(void) { return "fake"; }

static void fail(const char *what) { printf("%s: %zu rows of %zu bytes, at byte %zu\n", what, g_rows, g_row_bytes, g_at); exit(1); }

int spgk_memcpy_h2d(void *d, const void *h, size_t bytes, void *s)
{
    (void)s;
    if (g_in) {
        if (!bytes || ++g_copies > 64) fail("a copy of nothing");
        if (g_at + bytes > g_rows * g_row_bytes || memcmp(h, (const char *)g_in + g_at, bytes) != 0) fail("wrong rows staged");
        const size_t chunk = g_at / g_row_bytes / CHUNK, rows = g_rows - chunk * CHUNK < CHUNK ? g_rows - chunk * CHUNK : CHUNK;
        if (bytes != rows * g_row_bytes && bytes < (size_t)4 << 20) fail("a piece for one thread");
        g_at += bytes;
    }
    memcpy(d, h, bytes);
    return 0;
}

int main(void)
{
    spingalett_set_verbose(false);
    static const uint32_t tails[] = { 1, 2, 7, 8, 9, 15, 16, 17, 1234, 16383, 16384 }, widths[] = { 1, 20, 96, 128, 300 };
    for (size_t w = 0; w < sizeof widths / sizeof *widths; w++) {
        NeuralNetwork *net = new_spingalett();
        layer(.net = net, .neurons_amount = widths[w], .act_func = ACT_SIGMOID);
        layer(.net = net, .neurons_amount = 3, .act_func = ACT_SIGMOID);
        const size_t most = 3 * CHUNK;
        float *x = malloc(most * widths[w] * sizeof *x), *y = malloc(most * 3 * sizeof *y);
        for (size_t i = 0; i < most * widths[w]; i++) x[i] = (float)(i % 65521);
        for (size_t t = 0; t < sizeof tails / sizeof *tails; t++) {
            if (!forward_batch(.net = net, .inputs = x, .sample_count = 1, .outputs = y)) return 2;     /* uploads the net */
            g_rows = 2 * CHUNK + tails[t]; g_row_bytes = widths[w] * sizeof *x; g_at = 0; g_copies = 0; g_in = x;
            const float *r = forward_batch(.net = net, .inputs = x, .sample_count = (uint32_t)g_rows, .outputs = y);
            g_in = NULL;
            if (!r) { printf("%s\n", spingalett_last_error_message()); return 3; }
            if (g_at != g_rows * g_row_bytes) fail("rows missing");
        }
        free(x); free(y);
        free_network(net);
    }
    puts("all staged");
    return 0;
}
