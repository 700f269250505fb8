/* Outputs that lie where the inputs do: the kernels that read a batch's rows while they write others' outputs are not for such calls.  Host code of the
 * library on fake kernels, as in row_count.c. */
#include <stdio.h>
#include <stdlib.h>
#include <string.h>
#include "spingalett_b200.h"
#include "spingalett_b200_kernels.h"

static int g_whole, g_layers, g_rows, g_gemv;

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
int spgk_gemm_tc_softmax_fusable(uint32_t out, uint32_t N, int dynamic) { (void)out; (void)N; (void)dynamic; return 1; }
uint32_t spgk_gemm_tc_softmax_max(void) { return 1024; }
size_t spgk_weights16_bytes(const spgk_layer *L, int parts) { (void)L; (void)parts; return 256; }
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
    (void)y; (void)ldy; (void)softmax_fused; (void)weights_ready; (void)scratch; (void)status; (void)stream;
    g_whole++;
    return 0;
}
int spgk_layer_gemm_tc(const spgk_layer *L, const void *w16, uint32_t ldw, uint64_t w_plane, int w_parts, int w_type16, const void *a16, uint32_t lda,
                       uint64_t a_plane, int a_parts, int type16, void *out16, uint32_t ldo16, uint64_t o_plane, int out_parts, float *out32, uint32_t ldo32,
                       uint32_t N, int softmax_fused, int32_t *status, void *stream)
{
    (void)L; (void)w16; (void)ldw; (void)w_plane; (void)w_parts; (void)w_type16; (void)a16; (void)lda; (void)a_plane; (void)a_parts; (void)type16; (void)out16;
    (void)ldo16; (void)o_plane; (void)out_parts; (void)out32; (void)ldo32; (void)N; (void)softmax_fused; (void)status; (void)stream;
    g_layers++;
    return 0;
}
int spgk_rows_forward(const spgk_layer *layers, uint32_t count, const float *x, uint32_t ldx, float *const *ys, uint32_t N, void *stream)
{
    (void)layers; (void)count; (void)x; (void)ldx; (void)ys; (void)N; (void)stream;
    g_rows++;
    return 0;
}
int spgk_layer_gemv_chain(const spgk_layer *L, const spgk_layer *next, const void *staged, void *next_staged, const float *x, uint32_t ldx, float *y, uint32_t ldy,
                          uint32_t N, void *scratch, void *stream)
{
    (void)L; (void)next; (void)staged; (void)next_staged; (void)x; (void)ldx; (void)y; (void)ldy; (void)N; (void)scratch; (void)stream;
    g_gemv++;
    return 0;
}

static void expect(const char *what, NeuralNetwork *net, const float *x, uint32_t rows, float *y, int whole, int layers, int small, int gemv)
{
    g_whole = g_layers = g_rows = g_gemv = 0;
    if (!forward_batch(.net = net, .inputs = x, .sample_count = rows, .outputs = y)) { puts(spingalett_last_error_message()); exit(2); }
    if (g_whole != whole || g_layers != layers || g_rows != small || g_gemv != gemv) {
        printf("%s: %d whole, %d layers, %d small, %d gemv\n", what, g_whole, g_layers, g_rows, g_gemv);
        exit(1);
    }
}

int main(void)
{
    static float memory[700 * 16 + 700 * 8];
    float *const x = memory, *const y = memory + 700 * 16;
    spingalett_set_verbose(false);
    spingalett_set_math_mode(SPINGALETT_MATH_EXACT);
    NeuralNetwork *net = new_spingalett();
    layer(.net = net, .neurons_amount = 16);
    layer(.net = net, .neurons_amount = 24, .act_func = ACT_RELU);
    layer(.net = net, .neurons_amount = 8, .act_func = ACT_SIGMOID);
    expect("apart", net, x, 700, y, 1, 0, 0, 0);
    expect("one behind the other", net, x, 700, x + 700 * 16, 1, 0, 0, 0);
    expect("same place", net, x, 700, x, 0, 2, 0, 0);
    expect("last input", net, x, 700, x + 700 * 16 - 1, 0, 2, 0, 0);
    expect("last output", net, x + 700 * 8 - 1, 700, x, 0, 2, 0, 0);
    expect("a few rows", net, x, 4, x, 0, 0, 1, 0);            /* (the input is read by the first layer alone) */
    free_network(net);
    net = new_spingalett();
    layer(.net = net, .neurons_amount = 16);
    layer(.net = net, .neurons_amount = 8, .act_func = ACT_TANH);
    expect("one layer, apart", net, x, 4, y, 0, 0, 1, 0);
    expect("one layer, same place", net, x, 4, x, 0, 0, 0, 1);
    free_network(net);
    puts("every call on its kernel");
    return 0;
}
