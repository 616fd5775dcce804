// A device of FAKE_BYTES bytes with one context at a time, for the block cache's
// tests without a GPU: the runtime and driver calls csrc/block_cache.cu makes,
// counting what is allocated.  A call the device refuses returns its error.
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>

#include <cuda.h>
#include <cuda_runtime.h>

#include "block_cache.hpp"

extern "C" int lulesh_release_memory(void);

static const size_t kDeviceBytes = size_t(1) << 30;
static std::map<char *, size_t> g_live[2];  // device, pinned
static size_t g_used[2];
static int g_mallocs, g_wrong_frees;
static bool g_context = false, g_id_fails = false;
static unsigned long long g_id = 0;
static char *g_next = (char *)0x10000;

static cudaError_t fake_malloc(void **p, size_t n, int pinned)
{
    if (!g_context) g_context = true, ++g_id;
    ++g_mallocs;
    if (!pinned && g_used[0] + n > kDeviceBytes) return cudaErrorMemoryAllocation;
    *p = g_next;
    g_next += (n + 511) / 512 * 512 + 512;
    g_live[pinned][(char *)*p] = n;
    g_used[pinned] += n;
    return cudaSuccess;
}

static cudaError_t fake_free(void *p, int pinned)
{
    if (!g_context) g_context = true, ++g_id;
    if (!p) return cudaSuccess;
    auto it = g_live[pinned].find((char *)p);
    if (it == g_live[pinned].end()) return ++g_wrong_frees, cudaErrorInvalidValue;
    g_used[pinned] -= it->second;
    g_live[pinned].erase(it);
    return cudaSuccess;
}

static void reset()  // cudaDeviceReset
{
    g_context = false;
    for (int k = 0; k < 2; ++k) g_live[k].clear(), g_used[k] = 0;
    g_next = (char *)0x10000;  // the same addresses again
}

static CUresult current(CUcontext *c)
{
    *c = g_id ? (CUcontext)0x1 : nullptr;
    return CUDA_SUCCESS;
}
static CUresult context_id(CUcontext, unsigned long long *id)
{
    if (!g_context || g_id_fails) return CUDA_ERROR_CONTEXT_IS_DESTROYED;
    *id = g_id;
    return CUDA_SUCCESS;
}

extern "C" {
cudaError_t cudaGetDevice(int *d) { return *d = 0, cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetLastError(void) { return cudaSuccess; }
cudaError_t cudaMalloc(void **p, size_t n) { return fake_malloc(p, n, 0); }
cudaError_t cudaMallocHost(void **p, size_t n) { return fake_malloc(p, n, 1); }
cudaError_t cudaFree(void *p) { return fake_free(p, 0); }
cudaError_t cudaFreeHost(void *p) { return fake_free(p, 1); }
cudaError_t cudaGetDriverEntryPoint(const char *name, void **f, unsigned long long,
                                    cudaDriverEntryPointQueryResult *q)
{
    *f = !std::strcmp(name, "cuCtxGetCurrent") ? (void *)current
         : !std::strcmp(name, "cuCtxGetId")    ? (void *)context_id
                                               : nullptr;
    *q = *f ? cudaDriverEntryPointSuccess : cudaDriverEntryPointSymbolNotFound;
    return cudaSuccess;
}
}

#define CHECK(c)                                                          \
    do {                                                                  \
        if (!(c)) {                                                       \
            std::printf("line %d: %s\n", __LINE__, #c);                   \
            return 1;                                                     \
        }                                                                 \
    } while (0)

using namespace lulesh;
static const size_t MB = size_t(1) << 20;

int main()
{
    Block a, b, c;
    // a closed set's block is the next one's, and at most 512 MB are kept
    CHECK(block_get(&a, 300 * MB) == cudaSuccess);
    void *p = a.p;
    block_put(&a);
    CHECK(a.p == nullptr && g_used[0] == 300 * MB);
    CHECK(block_get(&a, 300 * MB) == cudaSuccess && a.p == p && g_mallocs == 1);
    CHECK(block_get(&b, 300 * MB) == cudaSuccess);
    block_put(&a);
    block_put(&b);
    CHECK(g_used[0] == 300 * MB);
    // a smaller set gets it, but never half empty
    CHECK(block_get(&a, 270 * MB) == cudaSuccess && a.p == p && a.bytes == 300 * MB);
    block_put(&a);
    CHECK(block_get(&a, 140 * MB) == cudaSuccess && a.p != p);
    block_free(&a);
    // and beyond an eighth only while all in use waste 128 MB at most
    CHECK(block_get(&a, 170 * MB) == cudaSuccess && a.p != p);
    block_free(&a);
    CHECK(block_get(&a, 200 * MB) == cudaSuccess && a.p == p);
    CHECK(block_get(&b, 200 * MB) == cudaSuccess);
    block_put(&b);
    CHECK(block_get(&b, 150 * MB) == cudaSuccess && b.bytes == 150 * MB);
    block_put(&b);
    CHECK(block_get(&b, 185 * MB) == cudaSuccess && b.bytes == 200 * MB);
    block_free(&b);
    lulesh_release_memory();
    block_put(&a);
    CHECK(g_used[0] == 300 * MB);
    CHECK(block_get(&a, 200 * MB) == cudaSuccess && a.p == p);
    block_put(&a);
    // a block from the driver instead of the cache wastes nothing
    CHECK(block_get(&a, 172 * MB) == cudaSuccess && a.p == p);
    block_put(&a);
    // block_free keeps nothing
    CHECK(block_get(&a, 300 * MB) == cudaSuccess && a.p == p);
    block_free(&a);
    CHECK(a.p == nullptr && g_used[0] == 0);

    // an allocation that does not fit beside what is kept gets that first:
    // through the cache, past it, and any other call
    CHECK(block_get(&a, 500 * MB) == cudaSuccess);
    block_put(&a);
    CHECK(block_get(&b, 800 * MB) == cudaSuccess && g_used[0] == 800 * MB);
    block_put(&b);
    CHECK(g_used[0] == 0);
    CHECK(block_get(&a, 500 * MB) == cudaSuccess);
    block_put(&a);
    void *q = nullptr;
    CHECK(device_malloc(&q, 800 * MB) == cudaSuccess && g_used[0] == 800 * MB);
    CHECK(cudaFree(q) == cudaSuccess);
    CHECK(block_get(&a, 500 * MB) == cudaSuccess);
    block_put(&a);
    CHECK(retry_trimmed([&] { return cudaMalloc(&q, 900 * MB); }) == cudaSuccess);
    CHECK(cudaFree(q) == cudaSuccess);
    // what does not fit at all is refused, after one more try at most
    CHECK(block_get(&a, 100 * MB) == cudaSuccess);
    block_put(&a);
    g_mallocs = 0;
    CHECK(device_malloc(&q, 2048 * MB) == cudaErrorMemoryAllocation && g_mallocs == 2);
    CHECK(device_malloc(&q, 2048 * MB) == cudaErrorMemoryAllocation && g_mallocs == 3);
    CHECK(block_get(&a, 2048 * MB) == cudaErrorMemoryAllocation && !a.p);

    // the program asks for it
    CHECK(block_get(&a, 400 * MB) == cudaSuccess && block_get(&b, 4096, true) == cudaSuccess);
    block_put(&a);
    block_put(&b);
    CHECK(g_used[0] == 400 * MB && g_used[1] == 4096);
    CHECK(lulesh_release_memory() == 0 && g_used[0] == 0 && g_used[1] == 0);
    CHECK(!block_trim());

    // a context's id that cannot be read: nothing is kept, nothing is lost
    CHECK(block_get(&a, 200 * MB) == cudaSuccess);
    p = a.p;
    block_put(&a);
    g_id_fails = true;
    CHECK(block_get(&b, 200 * MB) == cudaSuccess && b.p != p);
    block_put(&b);
    CHECK(g_used[0] == 200 * MB);
    g_id_fails = false;
    CHECK(block_get(&a, 200 * MB) == cudaSuccess && a.p == p);
    block_put(&a);

    // a device reset takes what is kept; a block from before it is not kept
    CHECK(block_get(&c, 100 * MB) == cudaSuccess);
    reset();
    CHECK(block_get(&a, 200 * MB) == cudaSuccess && g_used[0] == 200 * MB);
    CHECK(g_live[0].count((char *)a.p) == 1 && g_live[0].size() == 1);
    block_put(&a);
    block_put(&c);  // as cudaFree on an ended context's pointer: its address may be another's
    CHECK(g_wrong_frees <= 1);

    // many small blocks: 64 are kept
    lulesh_release_memory();
    Block many[100];
    const size_t before = g_used[0];
    for (Block &m : many) CHECK(block_get(&m, 8192) == cudaSuccess);
    for (Block &m : many) block_put(&m);
    CHECK(g_used[0] - before == 64 * 8192);
    std::printf("BLOCKS_OK\n");
    return 0;
}
