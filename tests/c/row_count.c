/* The device-resident number of rows that an AUTO call recomputes is zero when the call starts to list rows, whatever came before: a batch
 * that outgrows the list (whose memory the allocator may hand out at the same address, with other contents), a call that failed half way, a
 * captured call and its replays between direct ones, a net whose device state was dropped.  Rows are listed without a bound, so a count that
 * starts elsewhere is a write beyond the list.  Host code of the library on fake kernels, as in unread_status.c; freed "device memory" is the
 * next to be handed out and is full of something else. */
#include <stdio.h>
#include <stdlib.h>
#include <string.h>
#include "spingalett_b200.h"
#include "spingalett_b200_kernels.h"

#define BLOCK ((size_t)1 << 20)
static void *g_free[64];
static int g_free_count, g_fail_at, g_gemms, g_capturing, g_recorded;
static uint32_t g_list_rows;                   /* rows that a pass lists */
static uint32_t *g_idx, *g_count, *g_rows;     /* margin sink, and the count of the recomputation */

int spgk_device_count(int *n) { *n = 1; return 0; }
int spgk_get_device(int *d) { *d = 0; return 0; }
int spgk_malloc(void **p, size_t bytes)
{
    if (bytes > BLOCK) exit(20);
    *p = g_free_count ? g_free[--g_free_count] : malloc(BLOCK);
    memset(*p, 0x5A, BLOCK);
    return 0;
}
int spgk_free(void *p) { if (p) g_free[g_free_count++] = p; return 0; }
int spgk_host_alloc(void **p, size_t bytes) { *p = malloc(bytes); return 0; }
int spgk_host_free(void *p) { free(p); return 0; }
int spgk_memcpy_h2d(void *d, const void *h, size_t bytes, void *s) { (void)s; memcpy(d, h, bytes); return 0; }
int spgk_memcpy_d2h(void *h, const void *d, size_t bytes, void *s) { (void)s; memcpy(h, d, bytes); return 0; }
int spgk_is_device_pointer(const void *p) { (void)p; return 1; }
const char *spgk_error_string(void) { return "fake"; }
int spgk_gemm_tc_supported(const spgk_layer *L) { (void)L; return 1; }
int spgk_gemm_tc_softmax_fusable(uint32_t out, uint32_t N, int dynamic) { (void)out; (void)N; (void)dynamic; return 1; }
uint32_t spgk_gemm_tc_softmax_max(void) { return 1024; }
size_t spgk_weights16_bytes(const spgk_layer *L, int parts) { (void)L; (void)parts; return 256; }
void spgk_set_margin_sink(float theta, uint32_t *idx, uint32_t *count) { (void)theta; g_idx = idx; g_count = count; }
void spgk_set_dynamic_rows(const uint32_t *count, uint32_t expected) { (void)expected; g_rows = (uint32_t *)count; }
int spgk_stream_capturing(void *s) { (void)s; return g_capturing; }

static void list_rows(uint32_t *count)
{
    if (*count != 0) { printf("the count starts at %u\n", *count); exit(1); }
    *count = g_list_rows;
}

/* what is captured runs when the graph is launched */
static uint32_t *g_graph_clear, *g_graph_count, *g_graph_host;
static void replay(void)
{
    if (g_graph_clear) *g_graph_clear = 0;
    list_rows(g_graph_count);
    *g_graph_host = *g_graph_count;
    *g_graph_count = 0;
}

int spgk_memset(void *p, int v, size_t bytes, void *s)
{
    (void)s;
    if (g_capturing) { if (bytes == 4) g_graph_clear = p; return 0; }
    memset(p, v, bytes);
    return 0;
}

int spgk_layer_gemm_tc(const spgk_layer *L, const void *w16, uint32_t ldw, uint64_t w_plane, int w_parts, int w_type16, const void *a16, uint32_t lda,
                       uint64_t a_plane, int a_parts, int type16, void *out16, uint32_t ldo16, uint64_t o_plane, int out_parts, float *out32, uint32_t ldo32,
                       uint32_t N, int softmax_fused, int32_t *status, void *stream)
{
    (void)w16; (void)ldw; (void)w_plane; (void)w_parts; (void)w_type16; (void)a16; (void)lda; (void)a_plane; (void)a_parts; (void)type16; (void)out16;
    (void)ldo16; (void)o_plane; (void)out_parts; (void)out32; (void)ldo32; (void)N; (void)softmax_fused; (void)status; (void)stream;
    if (++g_gemms == g_fail_at) return SPGK_E_CUDA;
    if (g_count && L->act == ACT_SOFTMAX) {
        if (g_capturing) g_graph_count = g_count;
        else list_rows(g_count);
    }
    return 0;
}
int spgk_margin_select(const float *probs, uint32_t ldp, uint32_t N, uint32_t width, float theta, uint32_t *idx, uint32_t *count, void *stream)
{
    (void)probs; (void)ldp; (void)N; (void)width; (void)theta; (void)idx; (void)stream;
    list_rows(count);
    return 0;
}
int spgk_gap_error(const float *a, const float *b, uint32_t ld, uint32_t rows, uint32_t width, uint32_t *max_bits, void *stream)
{
    (void)a; (void)b; (void)ld; (void)rows; (void)width; (void)stream;
    *max_bits = 0x3C000000;
    return 0;
}
int spgk_count_take(uint32_t *count, uint32_t *host, void *stream)
{
    (void)stream;
    if (g_capturing) { g_graph_host = host; g_recorded = 1; return 0; }
    *host = *count;
    *count = 0;
    return 0;
}

static NeuralNetwork *g_net;
static float g_x[4096 * 8], g_y[4096 * 4];
static void call(uint32_t rows, uint32_t listed)
{
    g_list_rows = listed;
    if (!forward_batch(.net = g_net, .inputs = g_x, .sample_count = rows, .outputs = g_y)) { puts(spingalett_last_error_message()); exit(2); }
    if (spingalett_last_repaired(g_net) != listed) { printf("%u rows listed, %u reported\n", listed, spingalett_last_repaired(g_net)); exit(3); }
}

int main(void)
{
    spingalett_set_verbose(false);
    spingalett_set_math_mode(SPINGALETT_MATH_AUTO);
    g_net = new_spingalett();
    layer(.net = g_net, .neurons_amount = 8);
    layer(.net = g_net, .neurons_amount = 16, .act_func = ACT_RELU);
    layer(.net = g_net, .neurons_amount = 4, .act_func = ACT_SOFTMAX);
    for (int margin = 0; margin < 2; margin++) {
        spingalett_set_auto_margin(margin ? 0.5f : 0.0f);            /* measured on the first call, and given */
        for (uint32_t rows = 600; rows < 4000; rows += 500) { call(rows, rows / 9); call(600, 5); }
        /* a call that fails after its rows were listed: in the recomputation, and in a pass */
        for (int at = 1; at <= 4; at++) {
            g_gemms = 0; g_fail_at = at; g_list_rows = 77;
            if (forward_batch(.net = g_net, .inputs = g_x, .sample_count = 700, .outputs = g_y)) return 4;
            spingalett_clear_error();
            g_fail_at = 0;
            call(700, 3);
        }
        /* captured after a direct call and after a failed one; replayed between direct calls */
        for (int failed = 0; failed < 2; failed++) {
            if (failed) {
                g_gemms = 0; g_fail_at = 4; g_list_rows = 77;
                if (forward_batch(.net = g_net, .inputs = g_x, .sample_count = 700, .outputs = g_y)) return 5;
                spingalett_clear_error();
                g_fail_at = 0;
            }
            g_graph_clear = g_graph_count = g_graph_host = NULL; g_recorded = 0;
            if (margin) {                                            /* (a margin that is known: nothing to wait for) */
                g_capturing = 1;
                if (!forward_batch(.net = g_net, .inputs = g_x, .sample_count = 700, .outputs = g_y)) return 6;
                g_capturing = 0;
                if (!g_recorded || !g_graph_count) return 7;
                replay(); replay();
                call(700, 9);
                *g_graph_count = 0x5A5A; replay();                   /* (a replay that was cut off: the next clears the count itself) */
                call(650, 2);
                replay();
            }
            call(700, 1);
        }
        spingalett_sync_weights(g_net);
    }
    free_network(g_net);
    puts("every count from zero");
    return 0;
}
