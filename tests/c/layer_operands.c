/* The streaming kernel writes the next layer's operand only for a layer that it serves itself, into a buffer that has room for it: a net whose
 * layers go to the GEMV and to the streaming kernel by turns, in every pattern, at 1 to 8 rows.  Host code of the library on fake
 * kernels, as in unread_status.c; "device memory" is the heap with its length in front. */
#include <stdio.h>
#include <stdlib.h>
#include <string.h>
#include "spingalett_b200.h"
#include "spingalett_b200_kernels.h"

static const uint32_t g_widths[] = { 64, 65536, 160, 96, 32 };       /* (more weights than the kernel for small nets takes) */
#define LAYERS 4
static unsigned g_gemv;                        /* bit l: the GEMV takes layer l */
static const void *g_written;                  /* the operand that the layer before wrote */

int spgk_device_count(int *n) { *n = 1; return 0; }
int spgk_get_device(int *d) { *d = 0; return 0; }
int spgk_malloc(void **p, size_t bytes)
{
    size_t *b = malloc(16 + bytes);
    *b = bytes;
    *p = b + 2;
    return 0;
}
int spgk_free(void *p) { if (p) free((size_t *)p - 2); return 0; }
static size_t room(const void *p) { return p ? ((const size_t *)p)[-2] : 0; }
int spgk_is_device_pointer(const void *p) { (void)p; return 1; }
const char *spgk_error_string(void) { return "fake"; }

static int number(const spgk_layer *L) { for (int l = 0; l < LAYERS; l++) if (L->in == g_widths[l] && L->out == g_widths[l + 1]) return l; exit(20); }
size_t spgk_gemv_scratch_bytes(const spgk_layer *L, uint32_t N) { return N <= SPGK_GEMV_MAX_BATCH && (g_gemv >> number(L) & 1u) ? 64 : 0; }
size_t spgk_gemv_staged_bytes(uint32_t width, uint32_t N) { return (size_t)width * N; }
int spgk_gemv_forward_chain(const spgk_layer *L, uint32_t count, const float *x, uint32_t ldx, float *const *ys, uint32_t N, void *a, void *b, void *scratch, void *s)
{
    (void)L; (void)count; (void)x; (void)ldx; (void)ys; (void)N; (void)a; (void)b; (void)scratch; (void)s;
    return SPGK_E_UNSUPPORTED;
}
int spgk_layer_gemv_chain(const spgk_layer *L, const spgk_layer *next, const void *in, void *out, const float *x, uint32_t ldx, float *y, uint32_t ldy,
                          uint32_t N, void *scratch, void *s)
{
    (void)next; (void)in; (void)out; (void)x; (void)ldx; (void)y; (void)ldy; (void)s;
    if (!spgk_gemv_scratch_bytes(L, N)) return SPGK_E_UNSUPPORTED;
    if (room(scratch) < 64) exit(21);
    g_written = NULL;
    return 0;
}
size_t spgk_wstream_scratch_bytes(const spgk_layer *L, uint32_t N) { (void)L; (void)N; return 64; }
size_t spgk_wstream_operand_bytes(uint32_t width, uint32_t N) { return (size_t)width * N * 4; }
int spgk_wstream_stages_next(const spgk_layer *L, const spgk_layer *next, uint32_t N) { (void)L; (void)N; return next != NULL; }
int spgk_layer_wstream(const spgk_layer *L, const spgk_layer *next, const void *in, void *out, const float *x, uint32_t ldx, float *y, uint32_t ldy,
                       uint32_t N, void *scratch, void *s)
{
    (void)x; (void)ldx; (void)y; (void)ldy; (void)s;
    if (room(scratch) < 64) exit(22);
    if (in && in != g_written) { printf("layer %d reads an operand that nobody wrote\n", number(L)); exit(1); }
    g_written = NULL;
    if (next && out) {
        if (room(out) < spgk_wstream_operand_bytes(next->in, N)) { printf("layer %d: %zu bytes for an operand of %u\n", number(L), room(out), next->in); exit(1); }
        if (spgk_gemv_scratch_bytes(next, N)) { printf("layer %d writes an operand that nobody reads\n", number(L)); exit(1); }
        g_written = out;
    }
    return 0;
}

int main(void)
{
    spingalett_set_verbose(false);
    static float x[8 * 64], y[8 * 32];
    for (g_gemv = 0; g_gemv < 1u << LAYERS; g_gemv++) {
        NeuralNetwork *net = new_spingalett();
        for (int l = 0; l <= LAYERS; l++) layer(.net = net, .neurons_amount = g_widths[l], .act_func = ACT_RELU, .weight_initialization = WEIGHT_INITIALIZATION_NONE);
        for (uint32_t rows = 1; rows <= 8; rows++)
            if (!forward_batch(.net = net, .inputs = x, .sample_count = rows, .outputs = y) || spingalett_synchronize(net)) { puts(spingalett_last_error_message()); return 2; }
        free_network(net);
    }
    puts("every operand fits");
    return 0;
}
