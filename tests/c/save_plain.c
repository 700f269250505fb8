/* A saved file is written without room reserved for it beforehand: file systems that allocate late then write out a file that replaces
 * another when it is closed, so that a model saved over an older one is not lost with it in a power cut a moment later; and a save that
 * fails leaves nothing behind but what it wrote.  Host code of the library on fake kernels, as in unread_status.c. */
#include <fcntl.h>
#include <stdio.h>
#include <stdlib.h>
#include "spingalett_b200.h"

static int g_reserved;
int fallocate(int fd, int mode, off_t at, off_t bytes) { (void)fd; (void)mode; (void)at; (void)bytes; g_reserved++; return 0; }
int posix_fallocate(int fd, off_t at, off_t bytes) { (void)fd; (void)at; (void)bytes; g_reserved++; return 0; }

int main(int argc, char **argv)
{
    if (argc < 2) return 2;
    spingalett_set_verbose(false);
    NeuralNetwork *net = new_spingalett();
    for (int l = 0; l < 3; l++) layer(.net = net, .neurons_amount = 1100, .act_func = ACT_RELU, .weight_initialization = WEIGHT_INITIALIZATION_NONE);
    for (int p = PRECISION_FLOAT32; p < PRECISION_COUNT; p++) save_spingalett(.net = net, .filename = argv[1], .precision = (PrecisionMode)p);
    free_network(net);
    puts(spingalett_last_error_code() ? spingalett_last_error_message() : g_reserved ? "room reserved" : "written");
    return 0;
}
