/* Callers of spg_bulk at the same time share the threads: prints how many the first one had, and how many the second had while the
 * first was at work and after it. */
#include <pthread.h>
#include <stdatomic.h>
#include <stdio.h>
#include <unistd.h>
#include "spg_internal.h"

static atomic_int first, in, done;

static void hold(void *ctx, size_t lo, size_t hi)
{
    (void)ctx; (void)lo; (void)hi;
    atomic_fetch_add(&first, 1);
    atomic_store(&in, 1);
    for (int i = 0; i < 20000 && !atomic_load(&done); i++) usleep(1000);
}
static void count(void *ctx, size_t lo, size_t hi) { (void)lo; (void)hi; atomic_fetch_add((atomic_int *)ctx, 1); }
static void *caller(void *arg) { spg_bulk(hold, arg, 1u << 20, 1, 1); return NULL; }

int main(void)
{
    atomic_int during = 0, after = 0;
    pthread_t t;
    if (pthread_create(&t, NULL, caller, NULL)) return 2;
    while (!atomic_load(&in)) usleep(1000);
    spg_bulk(count, &during, 1u << 20, 1, 1);
    atomic_store(&done, 1);
    pthread_join(t, NULL);
    spg_bulk(count, &after, 1u << 20, 1, 1);
    printf("%d %d %d\n", first, during, after);
    return 0;
}
