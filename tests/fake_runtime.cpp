// Stands in for the few CUDA runtime calls that the set-up and status entry points make, on host memory: remembers
// which memsets of the default stream the host has not waited for.  Preloaded in front of the real runtime.
#include <stdlib.h>
#include <string.h>

static int g_pending = 0, g_allocations = 0;
static void* g_allocation[16];
static unsigned char g_symbol[1 << 20];

extern "C" {
int fake_pending() { return g_pending; }
void* fake_allocation(int i) { return g_allocation[i]; }
int cudaMalloc(void** p, size_t n) { return g_allocation[g_allocations++ & 15] = *p = calloc(1, n), 0; }
int cudaFree(void* p) { return free(p), 0; }
int cudaMemset(void* p, int v, size_t n) { return memset(p, v, n), ++g_pending, 0; }
int cudaMemsetAsync(void* p, int v, size_t n, void* stream) { return memset(p, v, n), g_pending += stream == nullptr, 0; }
int cudaMemcpy(void* d, const void* s, size_t n, int) { return memcpy(d, s, n), g_pending = 0; }
int cudaDeviceSynchronize() { return g_pending = 0; }
int cudaStreamSynchronize(void* stream) { return g_pending = stream ? g_pending : 0, 0; }
int cudaGetDevice(int* d) { return *d = 0; }
int cudaGetSymbolAddress(void** p, const void*) { return *p = g_symbol, 0; }
int cudaEventCreate(void** e) { return *e = malloc(1), 0; }
int cudaEventDestroy(void* e) { return free(e), 0; }
}
