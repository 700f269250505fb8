/* train() where page-locked memory is short: the shuffled orders of the epochs arrive whole, each a permutation, and none is changed while it may
 * still be on its way.  Host code of the library on fake kernels, as in unread_status.c; a copy from page-locked memory happens when its stream is
 * waited for, or an event behind it. */
#include <stdio.h>
#include <stdlib.h>
#include <string.h>
#include "spingalett_b200.h"
#include "spingalett_b200_kernels.h"

#define SAMPLES 3000u
static size_t g_most;                          /* bytes of page-locked memory that can be had at a time */
static char *g_pinned[8]; static size_t g_pinned_bytes[8];
static const void *g_from; static void *g_to; static size_t g_bytes;      /* a copy under way */
static int g_orders;

int spgk_device_count(int *n) { *n = 1; return 0; }
int spgk_get_device(int *d) { *d = 0; return 0; }
int spgk_malloc(void **p, size_t bytes) { *p = calloc(1, bytes + 64); return 0; }
int spgk_free(void *p) { free(p); return 0; }
int spgk_host_alloc(void **p, size_t bytes)
{
    if (bytes > g_most) return SPGK_E_NOMEM;
    for (int i = 0; i < 8; i++)
        if (!g_pinned[i]) { *p = g_pinned[i] = malloc(bytes); g_pinned_bytes[i] = bytes; return 0; }
    return SPGK_E_NOMEM;
}
int spgk_host_free(void *p) { for (int i = 0; i < 8; i++) if (p && g_pinned[i] == p) g_pinned[i] = NULL; free(p); return 0; }
int spgk_event_create(void **e) { *e = malloc(1); return 0; }
int spgk_event_destroy(void *e) { free(e); return 0; }
int spgk_stream_create(void **s) { *s = malloc(1); return 0; }
int spgk_stream_destroy(void *s) { free(s); return 0; }
int spgk_is_device_pointer(const void *p) { (void)p; return 0; }
const char *spgk_error_string(void) { return "fake"; }
size_t spgk_train_state_bytes(void) { return 64; }
int spgk_graph_begin(void *s) { (void)s; return SPGK_E_UNSUPPORTED; }

static void look(const uint32_t *order)
{
    static char seen[SAMPLES];
    memset(seen, 0, sizeof seen);
    for (uint32_t i = 0; i < SAMPLES; i++) {
        if (order[i] >= SAMPLES || seen[order[i]]) { puts("no permutation"); exit(1); }
        seen[order[i]] = 1;
    }
    g_orders++;
}
static void land(void)
{
    if (!g_to) return;
    memcpy(g_to, g_from, g_bytes);
    if (g_bytes == SAMPLES * 4) look(g_to);
    g_to = NULL;
}
int spgk_memcpy_h2d(void *d, const void *h, size_t bytes, void *s)
{
    (void)s;
    land();
    g_to = d; g_from = h; g_bytes = bytes;
    for (int i = 0; i < 8; i++)
        if (g_pinned[i] && (const char *)h >= g_pinned[i] && (const char *)h < g_pinned[i] + g_pinned_bytes[i]) return 0;
    land();                                    /* pageable: the driver has taken it when the call returns */
    return 0;
}
int spgk_memcpy_d2h(void *h, const void *d, size_t bytes, void *s) { (void)s; land(); memcpy(h, d, bytes); return 0; }
int spgk_stream_sync(void *s) { (void)s; land(); return 0; }
int spgk_event_sync(void *e) { (void)e; land(); return 0; }

int main(void)
{
    spingalett_set_verbose(false);
    static float x[SAMPLES * 2], t[SAMPLES * 2];
    for (uint32_t i = 0; i < SAMPLES * 2; i++) x[i] = t[i] = (float)(i & 1);
    static const size_t most[] = { (size_t)1 << 30, 4096, 1024 };
    for (int m = 0; m < 3; m++) {
        g_most = most[m];
        NeuralNetwork *net = new_spingalett(.loss_func = LOSS_CROSS_ENTROPY);
        layer(.net = net, .neurons_amount = 2);
        layer(.net = net, .neurons_amount = 2, .act_func = ACT_SOFTMAX, .weight_initialization = WEIGHT_INITIALIZATION_NONE);
        for (int call = 0; call < 2; call++) {
            g_orders = 0;
            train(.net = net, .inputs = x, .targets = t, .sample_count = SAMPLES, .batch_size = 100, .epochs = 5, .training_strategy = STRATEGY_SMALL_BATCH,
                  .optimizer_type = OPTIMIZER_ADAM);
            if (spingalett_last_error_code()) { printf("%zu bytes: %s\n", g_most, spingalett_last_error_message()); return 2; }
            if (g_orders != 5) { printf("%d orders\n", g_orders); return 3; }
        }
        free_network(net);
    }
    puts("every order");
    return 0;
}
