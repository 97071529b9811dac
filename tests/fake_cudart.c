/* Stand-ins for a few calls of the CUDA runtime, preloaded into a test's child process:
 *  - while armed, the launch of a kernel whose name holds a given text is passed on
 *    with an empty grid, which the runtime refuses on the host
 *    (cudaErrorInvalidConfiguration): nothing reaches the device;
 *  - launches are counted by kernel, graph instantiations in all;
 *  - the last allocation of at most 16 bytes is remembered (a status word);
 *  - on demand, memory and memsets behave as badly as the runtime allows (fake_late).
 * Everything else goes through unchanged. */
#define _GNU_SOURCE
#include <dlfcn.h>
#include <string.h>

#include <cuda_runtime_api.h>

#define MAXK 512
static struct {
    const void *func;
    const char *name;
    int count;
} g_k[MAXK];
static int g_nk, g_skip, g_refused, g_graphs;
static char g_text[64];
static void *g_small;

/* Refuse every launch of the kernels named so but the first `skip` ("": none). */
void fake_arm(const char *text, int skip)
{
    strncpy(g_text, text, sizeof g_text - 1);
    g_skip = skip;
    g_refused = 0;
}

int fake_refused(void) { return g_refused; }

/* Launches of the kernels named so since the last fake_reset. */
int fake_count(const char *text)
{
    int n = 0;
    for (int i = 0; i < g_nk; i++)
        if (strstr(g_k[i].name, text)) n += g_k[i].count;
    return n;
}

int fake_graphs(void) { return g_graphs; }

void fake_reset(void)
{
    for (int i = 0; i < g_nk; i++) g_k[i].count = 0;
    g_graphs = 0;
}

void *fake_small(void) { return g_small; }

/* The runtime itself, already loaded by the library under test. */
static void *runtime(const char *name) { return dlsym(dlopen("libcudart.so.12", RTLD_NOLOAD | RTLD_NOW), name); }
#define REAL(name) if (!real) *(void **)&real = runtime(name)

/* A launch of `func`: counted; 1 to refuse it. */
static int seen(const void *func)
{
    static cudaError_t (*real)(const char **, const void *);
    int i = 0;
    REAL("cudaFuncGetName");
    while (i < g_nk && g_k[i].func != func) i++;
    if (i == g_nk) {
        const char *n = 0;
        if (g_nk == MAXK || real(&n, func) != cudaSuccess || !n) return 0;
        g_k[g_nk].func = func;
        g_k[g_nk++].name = n;
    }
    if (g_text[0] && strstr(g_k[i].name, g_text)) {
        if (g_skip-- <= 0) {
            g_refused++;
            return 1;
        }
    }
    g_k[i].count++;
    return 0;
}


cudaError_t cudaLaunchKernel(const void *func, dim3 grid, dim3 block, void **args, size_t smem, cudaStream_t st)
{
    static cudaError_t (*real)(const void *, dim3, dim3, void **, size_t, cudaStream_t);
    REAL("cudaLaunchKernel");
    if (seen(func)) grid.x = 0;
    return real(func, grid, block, args, smem, st);
}

cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t *config, const void *func, void **args)
{
    static cudaError_t (*real)(const cudaLaunchConfig_t *, const void *, void **);
    cudaLaunchConfig_t c = *config;
    REAL("cudaLaunchKernelExC");
    if (seen(func)) c.gridDim.x = 0;
    return real(&c, func, args);
}

cudaError_t cudaGraphInstantiate(cudaGraphExec_t *exec, cudaGraph_t graph, unsigned long long flags)
{
    static cudaError_t (*real)(cudaGraphExec_t *, cudaGraph_t, unsigned long long);
    REAL("cudaGraphInstantiate");
    g_graphs++;
    return real(exec, graph, flags);
}

/* With fake_late(1): new memory holds 0xFF bytes, and cudaMemset, which the host does
 * not wait for and which another stream does not follow, takes effect only at the next
 * cudaMemcpy or cudaDeviceSynchronize. */
static int g_late, g_nset;
static struct {
    void *p;
    int v;
    size_t n;
} g_set[64];

void fake_late(int on) { g_late = on; }

static cudaError_t set_now(void *p, int v, size_t n)
{
    static cudaError_t (*real)(void *, int, size_t);
    REAL("cudaMemset");
    return real(p, v, n);
}

static void settle(void)
{
    for (int i = 0; i < g_nset; i++) set_now(g_set[i].p, g_set[i].v, g_set[i].n);
    g_nset = 0;
}

cudaError_t cudaMalloc(void **p, size_t n)
{
    static cudaError_t (*real)(void **, size_t);
    static cudaError_t (*wait)(void);
    REAL("cudaMalloc");
    const cudaError_t e = real(p, n);
    if (e != cudaSuccess) return e;
    if (n <= 16) g_small = *p;
    if (g_late) {
        if (!wait) *(void **)&wait = runtime("cudaDeviceSynchronize");
        set_now(*p, 0xFF, n);
        wait();
    }
    return e;
}

cudaError_t cudaMemset(void *p, int v, size_t n)
{
    if (!g_late || g_nset == 64) return set_now(p, v, n);
    g_set[g_nset].p = p;
    g_set[g_nset].v = v;
    g_set[g_nset++].n = n;
    return cudaSuccess;
}

cudaError_t cudaMemcpy(void *dst, const void *src, size_t n, enum cudaMemcpyKind kind)
{
    static cudaError_t (*real)(void *, const void *, size_t, enum cudaMemcpyKind);
    REAL("cudaMemcpy");
    settle();
    return real(dst, src, n, kind);
}

cudaError_t cudaDeviceSynchronize(void)
{
    static cudaError_t (*real)(void);
    REAL("cudaDeviceSynchronize");
    settle();
    return real();
}
