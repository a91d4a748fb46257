// Runs kernel_fit (csrc/kernel_fit.cpp) against a stand-in for the CUDA runtime that keeps
// the shared-memory consent by device and kernel, as the runtime does.
#include <cstdio>
#include <map>
#include <string>
#include <utility>

#include <cuda_runtime_api.h>

#include "kernel_fit.h"

static int device = 0, calls = 0;  // the stand-in's current device
static std::map<std::pair<int, const void *>, int> consent;
static std::map<const void *, int> resident;

extern "C" {
cudaError_t CUDARTAPI cudaFuncSetAttribute(const void *f, enum cudaFuncAttribute a, int v)
{
    if (a == cudaFuncAttributeMaxDynamicSharedMemorySize) consent[{device, f}] = v;
    return cudaSuccess;
}
cudaError_t CUDARTAPI cudaOccupancyMaxActiveBlocksPerMultiprocessor(int *n, const void *f, int, size_t)
{
    ++calls;
    *n = resident[f];
    return cudaSuccess;
}
cudaError_t CUDARTAPI cudaOccupancyMaxActiveClusters(int *n, const void *f, const cudaLaunchConfig_t *c)
{
    ++calls;
    *n = 100 * resident[f] + (int)c->attrs[0].val.clusterDim.x;
    return cudaSuccess;
}
cudaError_t CUDARTAPI cudaGetLastError() { return cudaSuccess; }
const char *CUDARTAPI cudaGetErrorString(cudaError_t) { return ""; }
}

#define CHECK(x)                                          \
    do {                                                  \
        if (!(x)) {                                       \
            std::printf("line %d: %s\n", __LINE__, #x);   \
            return 1;                                     \
        }                                                 \
    } while (0)

int main()
{
    const int a = 0, b = 0;  // addresses stand for kernels
    resident[&a] = 2;
    resident[&b] = 3;
    CHECK(gu::kernel_fit(0, &a, 512, 72000, 228352) == 2);
    CHECK((consent[{0, &a}] == 228352));
    // another kernel of the same shape: its own consent and count
    CHECK(gu::kernel_fit(0, &b, 512, 72000, 228352) == 3);
    CHECK((consent[{0, &b}] == 228352));
    // the same kernel and shape on another device: consent there too
    device = 1;
    CHECK(gu::kernel_fit(1, &a, 512, 72000, 228352) == 2);
    CHECK((consent[{1, &a}] == 228352));
    // clusters apart from single CTAs
    CHECK(gu::kernel_fit(1, &a, 512, 72000, 228352, 16) == 216);
    CHECK(gu::kernel_fit(1, &a, 512, 72000, 228352, 8) == 208);
    // asked again: kept
    const int before = calls;
    device = 0;
    CHECK(gu::kernel_fit(0, &b, 512, 72000, 228352) == 3);
    CHECK(gu::kernel_fit(1, &a, 512, 72000, 228352, 8) == 208);
    CHECK(calls == before);
    return 0;
}
