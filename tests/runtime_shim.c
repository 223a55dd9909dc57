/* Stands before the CUDA runtime (LD_PRELOAD) in child processes of tests: a device that has less memory, guard
 * bytes behind every allocation, and a count of shared-memory limits that a later call lowered. */
#define _GNU_SOURCE
#include <dlfcn.h>
#include <pthread.h>
#include <stdlib.h>
#include <string.h>

enum { MOST = 1 << 16, GUARD = 4096, OUT_OF_MEMORY = 2, MAX_DYNAMIC_SHARED = 8, DEVICE_TO_HOST = 2 };
static struct { void *p; size_t n; } live[MOST];
static struct { const void *f; int v; } limits[4096];
static size_t used, peak, limit = (size_t)-1;
static int n_live, n_limits, lowered, overrun;
static pthread_mutex_t mu = PTHREAD_MUTEX_INITIALIZER;

static void *real(const char *name)
{
    void *h = dlopen("libcudart.so.13", RTLD_NOLOAD | RTLD_LAZY);
    void *f = h ? dlsym(h, name) : NULL;
    if (!f) abort();
    return f;
}

void shim_limit(size_t bytes) { limit = bytes; }
size_t shim_used(void) { return used; }
size_t shim_peak(void) { return peak; }
void shim_reset_peak(void) { peak = used; }
int shim_lowered(void) { return lowered; }
int shim_overrun(void) { return overrun; }

int cudaMalloc(void **p, size_t n)
{
    int (*f)(void **, size_t) = real("cudaMalloc"), (*set)(void *, int, size_t) = real("cudaMemset");
    pthread_mutex_lock(&mu);
    int e = used + n > limit || n_live == MOST ? OUT_OF_MEMORY : f(p, n + GUARD);
    if (e == 0) {
        set((char *)*p + n, 0xA5, GUARD);
        live[n_live].p = *p;
        live[n_live++].n = n;
        used += n;
        if (used > peak) peak = used;
    }
    pthread_mutex_unlock(&mu);
    return e;
}

int cudaFree(void *p)
{
    int (*f)(void *) = real("cudaFree"), (*sync)(void) = real("cudaDeviceSynchronize");
    int (*copy)(void *, const void *, size_t, int) = real("cudaMemcpy");
    pthread_mutex_lock(&mu);
    for (int i = 0; p && i < n_live; ++i)
        if (live[i].p == p) {
            unsigned char g[GUARD], want[GUARD];
            memset(want, 0xA5, GUARD);
            if (sync() == 0 && copy(g, (char *)p + live[i].n, GUARD, DEVICE_TO_HOST) == 0 && memcmp(g, want, GUARD)) ++overrun;
            used -= live[i].n;
            live[i] = live[--n_live];
            break;
        }
    pthread_mutex_unlock(&mu);
    return f(p);
}

int cudaFuncSetAttribute(const void *func, int attr, int value)
{
    int (*f)(const void *, int, int) = real("cudaFuncSetAttribute");
    if (attr == MAX_DYNAMIC_SHARED) {
        pthread_mutex_lock(&mu);
        int i = 0;
        while (i < n_limits && limits[i].f != func) ++i;
        if (i == n_limits && n_limits < 4096) limits[n_limits++].f = func;
        if (i < n_limits) {
            if (value < limits[i].v) ++lowered;
            limits[i].v = value;
        }
        pthread_mutex_unlock(&mu);
    }
    return f(func, attr, value);
}
