// block_cache.cu -- see block_cache.hpp.
#include "block_cache.hpp"

#include <map>
#include <mutex>
#include <vector>

namespace lulesh {

namespace {

// A mark in the module's own device memory.  A device reset loads the module
// again with 0 here, so what carries an older mark belongs to an ended context.
__device__ unsigned long long g_mark;

struct Kept {
    std::vector<Block> blocks;
    size_t bytes = 0;
};

struct Store {
    unsigned long long mark = 0;  // as written to the device's g_mark, 0 none
    Kept kept[2];                 // device memory, pinned memory
};

std::mutex g_mu;
unsigned long long g_marks = 0;

// by device; never destroyed, as the driver may be gone at exit
std::map<int, Store> &stores()
{
    static auto *s = new std::map<int, Store>;
    return *s;
}

void free_block(const Block &b)
{
    const cudaError_t e = b.pinned ? cudaFreeHost(b.p) : cudaFree(b.p);
    if (e != cudaSuccess) (void)cudaGetLastError();
}

// the mark on the current device; 0 also when it cannot be read
unsigned long long read_mark()
{
    unsigned long long mark = 0;
    if (cudaMemcpyFromSymbolAsync(&mark, g_mark, sizeof mark, 0, cudaMemcpyDeviceToHost,
                                  cudaStreamPerThread) != cudaSuccess ||
        cudaStreamSynchronize(cudaStreamPerThread) != cudaSuccess) {
        (void)cudaGetLastError();
        return 0;
    }
    return mark;
}

unsigned long long write_mark()
{
    const unsigned long long mark = ++g_marks;
    if (cudaMemcpyToSymbolAsync(g_mark, &mark, sizeof mark, 0, cudaMemcpyHostToDevice,
                                cudaStreamPerThread) != cudaSuccess ||
        cudaStreamSynchronize(cudaStreamPerThread) != cudaSuccess) {
        (void)cudaGetLastError();
        return 0;
    }
    return mark;
}

void release(Kept &k)
{
    for (const Block &b : k.blocks) free_block(b);
    k = Kept{};
}

}  // namespace

cudaError_t block_get(Block *b, size_t bytes, bool pinned)
{
    Block n;
    cudaError_t e = cudaGetDevice(&n.device);
    if (e != cudaSuccess) return e;
    std::lock_guard<std::mutex> lock(g_mu);
    Store &s = stores()[n.device];
    if (s.mark == 0 || read_mark() != s.mark) {
        s = Store{};  // nothing kept, or gone with its context
        s.mark = write_mark();
    }
    Kept &k = s.kept[pinned];
    // the smallest block that is large enough and not twice too large
    size_t best = k.blocks.size();
    for (size_t i = 0; i < k.blocks.size(); ++i)
        if (k.blocks[i].bytes >= bytes && k.blocks[i].bytes <= 2 * bytes + 4096 &&
            (best == k.blocks.size() || k.blocks[i].bytes < k.blocks[best].bytes))
            best = i;
    if (best < k.blocks.size()) {
        *b = k.blocks[best];
        k.bytes -= b->bytes;
        k.blocks.erase(k.blocks.begin() + (long)best);
        return cudaSuccess;
    }
    n.bytes = bytes;
    n.mark = s.mark;
    n.pinned = pinned;
    for (int attempt = 0; attempt < 2; ++attempt) {
        e = pinned ? cudaMallocHost(&n.p, bytes) : cudaMalloc(&n.p, bytes);
        if (e != cudaErrorMemoryAllocation || (s.kept[0].blocks.empty() && s.kept[1].blocks.empty()))
            break;
        (void)cudaGetLastError();
        release(s.kept[0]);
        release(s.kept[1]);
    }
    if (e == cudaSuccess) *b = n;
    return e;
}

void block_put(Block *b)
{
    if (!b->p) return;
    const Block was = *b;
    *b = Block{};
    int prev = -1;
    cudaGetDevice(&prev);
    if (prev != was.device) cudaSetDevice(was.device);
    bool keep = false;
    {
        std::lock_guard<std::mutex> lock(g_mu);
        Store &s = stores()[was.device];
        Kept &k = s.kept[was.pinned];
        keep = was.mark != 0 && was.mark == s.mark && k.blocks.size() < kCacheBlocks &&
               k.bytes + was.bytes <= (was.pinned ? kCachePinnedBytes : kCacheDeviceBytes) &&
               read_mark() == was.mark;
        if (keep) {
            k.blocks.push_back(was);
            k.bytes += was.bytes;
        }
    }
    if (!keep) free_block(was);
    if (prev >= 0 && prev != was.device) cudaSetDevice(prev);
}

void block_free(Block *b)
{
    if (b->p) free_block(*b);
    *b = Block{};
}

}  // namespace lulesh
