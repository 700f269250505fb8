/* A net in one launch is told that its weight operands are there only when none of them is made in front of it: not in the first call, nor where the kept
 * ones have another number of terms and are made again.  Host code of the library on fake kernels, as in row_count.c. */
#include <stdio.h>
#include <stdlib.h>
#include <string.h>
#include "spg_internal.h"

static int g_launches, g_ready, g_made;

int spgk_device_count(int *n) { *n = 1; return 0; }
int spgk_get_device(int *d) { *d = 0; return 0; }
int spgk_malloc(void **p, size_t bytes) { *p = calloc(1, bytes + 256); return *p ? 0 : SPGK_E_NOMEM; }
int spgk_free(void *p) { free(p); return 0; }
int spgk_host_alloc(void **p, size_t bytes) { *p = malloc(bytes); return 0; }
int spgk_host_free(void *p) { free(p); return 0; }
int spgk_memcpy_h2d(void *d, const void *h, size_t bytes, void *s) { (void)s; memcpy(d, h, bytes); return 0; }
int spgk_is_device_pointer(const void *p) { (void)p; return 1; }
const char *spgk_error_string(void) { return "fake"; }
int spgk_gemm_tc_supported(const spgk_layer *L) { (void)L; return 1; }
size_t spgk_weights16_bytes(const spgk_layer *L, int parts) { (void)L; (void)parts; return 256; }
int spgk_dequant16(const spgk_layer *L, void *dst, uint32_t ldw, uint64_t plane, int parts, int type16, void *stream)
{
    (void)L; (void)dst; (void)ldw; (void)plane; (void)parts; (void)type16; (void)stream;
    g_made++;
    return 0;
}
int spgk_chain_plan(const spgk_layer *layers, uint32_t count, uint32_t N, int w_parts, int a_parts, int softmax_fused, spgk_chain *plan)
{
    (void)layers; (void)count; (void)N; (void)w_parts; (void)a_parts; (void)softmax_fused;
    *plan = (spgk_chain){ .C = 2, .R = 16, .clusters = 1, .exchange_bytes = 256, .scratch_bytes = 512, .us = 1.0f, .layered_us = 2.0f };
    return 0;
}
int spgk_chain_forward(const spgk_chain *plan, const spgk_layer *layers, uint32_t count, const void *const *w16, const uint32_t *ldw, const uint64_t *w_plane,
                       int w_parts, int type16, int a_parts, const float *x, uint32_t ldx, const uint32_t *x_rows, uint32_t N, float *y, uint32_t ldy,
                       int softmax_fused, int weights_ready, void *scratch, int32_t *status, void *stream)
{
    (void)plan; (void)layers; (void)count; (void)w16; (void)ldw; (void)w_plane; (void)w_parts; (void)type16; (void)a_parts; (void)x; (void)ldx; (void)x_rows; (void)N;
    (void)y; (void)ldy; (void)softmax_fused; (void)scratch; (void)status; (void)stream;
    g_launches++;
    g_ready = weights_ready;
    return 0;
}

static float memory[700 * 24];
static void expect(const char *what, NeuralNetwork *net, int made, int ready)
{
    g_launches = g_made = 0;
    if (!forward_batch(.net = net, .inputs = memory, .sample_count = 700, .outputs = memory + 700 * 16)) { puts(spingalett_last_error_message()); exit(2); }
    if (g_launches != 1 || g_made != made || g_ready != ready) {
        printf("%s: %d launches, %d operands made, ready %d\n", what, g_launches, g_made, g_ready);
        exit(1);
    }
}

int main(void)
{
    spingalett_set_verbose(false);
    spingalett_set_math_mode(SPINGALETT_MATH_EXACT);
    NeuralNetwork *net = new_spingalett();
    layer(.net = net, .neurons_amount = 16);
    layer(.net = net, .neurons_amount = 24, .act_func = ACT_RELU);
    layer(.net = net, .neurons_amount = 8, .act_func = ACT_SIGMOID);
    expect("first", net, 2, 0);
    expect("second", net, 0, 1);
    spg_priv(net)->w16c_parts[SPGK_T_BF16][1] = 1;
    expect("an operand of one term", net, 1, 0);
    expect("made again", net, 0, 1);
    free_network(net);
    puts("only when they are there");
    return 0;
}
