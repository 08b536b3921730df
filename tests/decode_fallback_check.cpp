// Prints the kernel launches of decode calls on a system whose driver builds no tensor maps, against a stand-in for the
// CUDA runtime that launches nothing: grid, cluster size and dynamic shared memory, a line per launch.
//   decode_fallback_check <library>
#include <cuda_runtime_api.h>
#include <dlfcn.h>

#include <cstdint>
#include <cstdio>
#include <cstdlib>

#include "../include/rustorch_attn.h"

// ---- the stand-in
extern "C" {
cudaError_t cudaGetDevice(int* d) { return *d = 0, cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr, int) { return *v = 148, cudaSuccess; }
cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute, int) { return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
cudaError_t cudaMemsetAsync(void*, int, size_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaGetSymbolAddress(void** p, const void*) { return *p = malloc(256), cudaSuccess; }
cudaError_t cudaGetDriverEntryPoint(const char*, void** p, unsigned long long, cudaDriverEntryPointQueryResult* r) {
    return *p = nullptr, *r = cudaDriverEntryPointSymbolNotFound, cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveClusters(int* n, const void*, const cudaLaunchConfig_t* c) {
    return *n = 128 / (int)c->attrs[0].val.clusterDim.x, cudaSuccess;
}
static cudaError_t launched(dim3 g, size_t smem, unsigned cluster) {
    return printf("grid %u %u %u cluster %u smem %zu\n", g.x, g.y, g.z, cluster, smem), cudaSuccess;
}
cudaError_t cudaLaunchKernel(const void*, dim3 g, dim3, void**, size_t smem, cudaStream_t) { return launched(g, smem, 1); }
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void*, void**) {
    unsigned cluster = 1;
    for (unsigned i = 0; i < c->numAttrs; ++i)
        if (c->attrs[i].id == cudaLaunchAttributeClusterDimension) cluster = c->attrs[i].val.clusterDim.x;
    return launched(c->gridDim, c->dynamicSmemBytes, cluster);
}
}

int main(int, char** argv) {
    void* lib = dlopen(argv[1], RTLD_NOW | RTLD_LOCAL);
    if (!lib) return fprintf(stderr, "%s\n", dlerror()), 1;
#define FN(name) auto* const name##_ = reinterpret_cast<decltype(&name)>(dlsym(lib, #name))
    FN(rt_gqa_decode_workspace_bytes);
    FN(rt_gqa_decode_bf16);
    FN(rt_gqa_decode_record_push_bf16);
    FN(rt_gqa_decode_exchange_bf16);
    // addresses that nothing reads
    auto at = [](uintptr_t a) { return reinterpret_cast<void*>(a << 20); };
    void* const slots[2] = {at(10), at(11)};
    void* const flags[2] = {at(12), at(13)};
    const struct { int64_t batch, n_kv; int dim; int64_t seq; bool ragged; } cases[] = {
        {1, 8, 128, 1000, false}, {1, 2, 256, 3000, false}, {1, 1, 64, 100, false}, {7, 2, 256, 3000, true}, {8, 8, 64, 1000, true}};
    for (const auto& c : cases) {
        const int64_t n_heads = 4 * c.n_kv;
        const size_t ws = rt_gqa_decode_workspace_bytes_(c.batch, n_heads, c.n_kv, c.dim, c.seq);
        const int32_t* lens = c.ragged ? static_cast<int32_t*>(at(14)) : nullptr;
        printf("batch %d KV heads %d D %d seq %d\n", (int)c.batch, (int)c.n_kv, c.dim, (int)c.seq);
        const int a = rt_gqa_decode_bf16_(at(1), at(2), at(3), at(4), nullptr, nullptr, c.batch, n_heads, c.n_kv, c.dim, c.seq, lens,
                                          c.seq, 0, -1, -1.f, at(5), ws, nullptr);
        const int b = rt_gqa_decode_record_push_bf16_(at(1), at(2), at(3), (float*)at(6), slots, flags, 2, 1, (int*)at(7), c.batch, n_heads,
                                                      c.n_kv, c.dim, c.seq, lens, c.seq, 0, -1, -1.f, at(5), ws, nullptr);
        const int d = rt_gqa_decode_exchange_bf16_(at(1), at(2), at(3), at(4), nullptr, nullptr, slots, flags, (const float*)slots[0],
                                                   (const uint32_t*)flags[0], 2, 0, 1, 0, 1, c.batch, n_heads, c.n_kv, c.dim, c.seq, lens,
                                                   c.seq, 0, -1, -1.f, at(5), ws, nullptr);
        printf("status %d %d %d\n", a, b, d);
    }
    return 0;
}
