/* A net of very many layers on a thread with a small stack: every layer is launched once, each on what the one before wrote.  Host code of the
 * library on fake kernels, as in unread_status.c. */
#include <pthread.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>
#include "spingalett_b200.h"
#include "spingalett_b200_kernels.h"

#define LAYERS 40000
static const float *g_x;
static uint32_t g_layers;

int spgk_device_count(int *n) { *n = 1; return 0; }
int spgk_get_device(int *d) { *d = 0; return 0; }
int spgk_malloc(void **p, size_t bytes) { *p = malloc(bytes); return 0; }
int spgk_free(void *p) { free(p); return 0; }
int spgk_is_device_pointer(const void *p) { (void)p; return 1; }
const char *spgk_error_string(void) { return "fake"; }
int spgk_rows_forward(const spgk_layer *L, uint32_t count, const float *x, uint32_t ldx, float *const *ys, uint32_t N, void *s)
{
    (void)s;
    for (uint32_t l = 0; l < count; l++) {
        if (x != g_x || ldx != L[l].in || N != 3) return SPGK_E_ARG;
        g_x = x = ys[l];
        ldx = L[l].out;
        g_layers++;
    }
    return 0;
}

static void *work(void *net)
{
    static float x[3], y[3];
    g_x = x;
    if (!forward_batch(.net = net, .inputs = x, .sample_count = 3, .outputs = y)) puts(spingalett_last_error_message());
    else if (g_layers != LAYERS || g_x != y) printf("%u layers\n", g_layers);
    else puts("every layer");
    return NULL;
}

int main(void)
{
    spingalett_set_verbose(false);
    NeuralNetwork *net = new_spingalett();
    for (int l = 0; l <= LAYERS; l++) layer(.net = net, .neurons_amount = 1, .act_func = ACT_RELU, .weight_initialization = WEIGHT_INITIALIZATION_NONE);
    pthread_attr_t a;
    pthread_t t;
    pthread_attr_init(&a);
    pthread_attr_setstacksize(&a, 256 << 10);
    if (pthread_create(&t, &a, work, net)) return 2;
    pthread_join(t, NULL);
    free_network(net);
    return 0;
}
