// Chunk meshing when device memory is short: this program's cudaMalloc, which the library then calls, refuses
// what goes past a budget.  With room for the scratch of one chunk only, a call for six has to mesh them
// in smaller groups and give the same meshes; with less it has to fail, and work again with more.
// Prints "<n> failures".
#include <cuda_runtime.h>
#include <dlfcn.h>

#include <cstdio>
#include <map>
#include <mutex>
#include <thread>
#include <vector>

#include "FastNoise/FastNoise_C.h"

namespace {
std::mutex g_mu;
std::map<void*, size_t> g_live;
size_t g_used = 0, g_budget = ~size_t(0), g_refused = 0, g_peak = 0;
}  // namespace

extern "C" cudaError_t CUDARTAPI cudaMalloc(void** p, size_t size)
{
    static const auto real = reinterpret_cast<cudaError_t (*)(void**, size_t)>(dlsym(RTLD_NEXT, "cudaMalloc"));
    std::lock_guard<std::mutex> lk(g_mu);
    if (g_used + size > g_budget) {
        ++g_refused;
        return cudaErrorMemoryAllocation;
    }
    const cudaError_t e = real(p, size);
    if (e == cudaSuccess) {
        g_live[*p] = size;
        g_used += size;
        if (g_used > g_peak) g_peak = g_used;
    }
    return e;
}

extern "C" cudaError_t CUDARTAPI cudaFree(void* p)
{
    static const auto real = reinterpret_cast<cudaError_t (*)(void*)>(dlsym(RTLD_NEXT, "cudaFree"));
    std::lock_guard<std::mutex> lk(g_mu);
    const auto it = g_live.find(p);
    if (it != g_live.end()) {
        g_used -= it->second;
        g_live.erase(it);
    }
    return real(p);
}

namespace {

constexpr int kSize = 64, kChunks = 6, kVerts = 2 * kSize * kSize * kSize, kIndices = 4 * kSize * kSize * kSize;

struct Buffers {
    char* v = nullptr;
    unsigned* i = nullptr;
    fnChunkMesh mesh[kChunks];
    int rc = 0;
    std::vector<char> verts;
    std::vector<unsigned> indices;
};

// A call on a thread of its own, whose scratch is new and ends with it; `single`: chunk by chunk.
void run(const void* node, Buffers& b, bool single)
{
    std::thread([&] {
        int pos[3 * kChunks];
        for (int k = 0; k < kChunks; ++k) {
            pos[3 * k] = 64 * k;
            pos[3 * k + 1] = -32;
            pos[3 * k + 2] = 64 * (k % 2);
            b.mesh[k] = fnChunkMesh();
            b.mesh[k].vertices = reinterpret_cast<fnMeshVertex*>(b.v + (size_t)k * kVerts * 16);
            b.mesh[k].indices = b.i + (size_t)k * kIndices;
            b.mesh[k].vertexCapacity = kVerts;
            b.mesh[k].indexCapacity = kIndices;
        }
        cudaMemset(b.v, 0, (size_t)kChunks * kVerts * 16);
        cudaMemset(b.i, 0, (size_t)kChunks * kIndices * 4);
        b.rc = 0;
        if (single)
            for (int k = 0; k < kChunks; ++k)
                b.rc |= fnBuildChunkMeshDmc(node, kSize, pos[3 * k], pos[3 * k + 1], pos[3 * k + 2], 7, 0.0f, 0, &b.mesh[k], nullptr);
        else
            b.rc = fnBuildChunkMeshesDmc(node, kSize, kChunks, pos, 7, 0.0f, 0, b.mesh, nullptr);
        b.verts.resize((size_t)kChunks * kVerts * 16);
        b.indices.resize((size_t)kChunks * kIndices);
        cudaMemcpy(b.verts.data(), b.v, b.verts.size(), cudaMemcpyDeviceToHost);
        cudaMemcpy(b.indices.data(), b.i, b.indices.size() * 4, cudaMemcpyDeviceToHost);
    }).join();
}

bool same(const Buffers& a, const Buffers& b)
{
    bool ok = a.verts == b.verts && a.indices == b.indices;
    for (int k = 0; k < kChunks; ++k)
        ok = ok && a.mesh[k].vertexCount == b.mesh[k].vertexCount && a.mesh[k].indexCount == b.mesh[k].indexCount &&
             a.mesh[k].minAirY == b.mesh[k].minAirY && a.mesh[k].maxSolidY == b.mesh[k].maxSolidY && a.mesh[k].vertexCount > 0;
    return ok;
}

}  // namespace

int main()
{
    void* node = fnNewFromMetadata(6, 0);                        // Simplex: a surface in every chunk
    if (!node || !fnSetVariableFloat(node, 0, 40.0f)) { std::printf("setup failed\n"); return 1; }
    Buffers b, ref;
    void *v = nullptr, *i = nullptr;
    if (cudaMalloc(&v, (size_t)kChunks * kVerts * 16) != cudaSuccess || cudaMalloc(&i, (size_t)kChunks * kIndices * 4) != cudaSuccess) {
        std::printf("allocation failed\n");
        return 1;
    }
    b.v = ref.v = static_cast<char*>(v);
    b.i = ref.i = static_cast<unsigned*>(i);
    int failures = 0;
    run(node, ref, true);                                        // the program and the workspaces exist from here on
    failures += ref.rc != 0;
    const size_t before = g_used;
    g_peak = before;
    run(node, ref, true);
    const size_t one = g_peak - before;                          // what one chunk takes
    g_peak = before;
    run(node, b, false);
    const size_t all = g_peak - before;
    failures += b.rc != 0 || !same(b, ref) || all < 2 * one;
    for (const size_t room : {one + one / 16, 2 * one + one / 8, 3 * one}) {
        g_budget = before + room;
        g_refused = 0;
        run(node, b, false);
        if (b.rc != 0 || !same(b, ref) || g_refused == 0) {
            ++failures;
            std::printf("room for %.2f chunks: status %d, %zu refused\n", (double)room / (double)one, b.rc, g_refused);
        }
    }
    g_budget = before + one / 2;
    run(node, b, false);
    failures += b.rc != FN_ERR_CUDA;
    g_budget = ~size_t(0);
    run(node, b, false);
    failures += b.rc != 0 || !same(b, ref);
    std::printf("%d failures\n", failures);
    fnDeleteNodeRef(node);
    return failures == 0 ? 0 : 1;
}
