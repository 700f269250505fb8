/* A bounded wait that gave up in a device-to-device call is reported by the next call that has to replace the buffer its
 * status lies in.  Host code of the library on fake kernels (tests/test_host_abi.py writes a stub for every spgk_ function that
 * is not defined here): "device memory" is the heap, and the first istream call leaves a failure in its scratch. */
#include <stdio.h>
#include <stdlib.h>
#include <string.h>
#include "spingalett_b200.h"
#include "spingalett_b200_kernels.h"

static int g_calls;

int spgk_device_count(int *n) { *n = 1; return 0; }
int spgk_get_device(int *d) { *d = 0; return 0; }
int spgk_malloc(void **p, size_t bytes) { *p = malloc(bytes); return 0; }
int spgk_free(void *p) { free(p); return 0; }
int spgk_memset(void *p, int v, size_t bytes, void *s) { (void)s; memset(p, v, bytes); return 0; }
int spgk_memcpy_h2d(void *d, const void *h, size_t bytes, void *s) { (void)s; memcpy(d, h, bytes); return 0; }
int spgk_is_device_pointer(const void *p) { (void)p; return 1; }
int spgk_gemv_get_int_path(void) { return 1; }
const char *spgk_error_string(void) { return "fake"; }
size_t spgk_istream_scratch_bytes(const spgk_layer *L, uint32_t count, uint32_t N) { (void)L; (void)count; return 64 + N; }
int spgk_istream_forward(const spgk_layer *L, uint32_t count, const float *x, uint32_t ldx, float *const *ys, uint32_t N, void *scratch, void *s)
{
    (void)L; (void)count; (void)x; (void)ldx; (void)ys; (void)N; (void)s;
    if (g_calls++ == 0) *(int32_t *)scratch = 9;
    return 0;
}
int spgk_istream_status(void *scratch, void *s) { (void)s; return *(int32_t *)scratch ? SPGK_E_TIMEOUT : 0; }

int main(int argc, char **argv)
{
    NeuralNetwork *net = new_spingalett();
    layer(.net = net, .neurons_amount = 64, .act_func = ACT_SIGMOID);
    layer(.net = net, .neurons_amount = 64, .act_func = ACT_SIGMOID);
    save_spingalett(.net = net, .filename = argc > 1 ? argv[1] : "net.nn", .precision = PRECISION_INT8);
    free_network(net);
    net = load_spingalett(argv[1]);
    if (!net) return 2;
    static float x[96 * 64], y[96 * 64];
    if (!forward_batch(.net = net, .inputs = x, .sample_count = 8, .outputs = y)) return 3;       /* stream-ordered: not known yet */
    if (forward_batch(.net = net, .inputs = x, .sample_count = 96, .outputs = y)) { puts("failure lost"); return 1; }
    if (spingalett_last_error_code() != SPINGALETT_ERR_DEVICE || g_calls != 1) return 4;
    spingalett_clear_error();
    if (!forward_batch(.net = net, .inputs = x, .sample_count = 96, .outputs = y) || spingalett_synchronize(net)) return 5;      /* and that was it */
    free_network(net);
    puts("reported");
    return 0;
}
