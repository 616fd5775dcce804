// block_cache.cu -- see block_cache.hpp.
#include "block_cache.hpp"

#include <cuda.h>

#include <map>
#include <mutex>
#include <utility>
#include <vector>

#include "lulesh_b200.h"

namespace lulesh {

namespace {

struct Kept {
    std::vector<Block> blocks;
    size_t bytes = 0;
};

struct Store {
    Kept kept[2];  // device memory, pinned memory
};

std::mutex g_mu;

// by context.  What is kept of a context that has ended (cudaDeviceReset) went
// with it: its entry is never looked up again and holds a few host bytes.  Never
// destroyed, as the driver may be gone at exit.
std::map<unsigned long long, Store> &stores()
{
    static auto *s = new std::map<unsigned long long, Store>;
    return *s;
}

void free_block(const Block &b)
{
    const cudaError_t e = b.pinned ? cudaFreeHost(b.p) : cudaFree(b.p);
    if (e != cudaSuccess) (void)cudaGetLastError();
}

// The id of the current context, unique for the life of the process: a reset
// device has a new one.  0 where it cannot be had, and nothing is kept then.  No
// stream is touched, so that a caller may be capturing any of its own.
unsigned long long context_id()
{
    using GetCurrent = CUresult (*)(CUcontext *);
    using GetId = CUresult (*)(CUcontext, unsigned long long *);
    struct Entry {
        GetCurrent current = nullptr;
        GetId id = nullptr;
        Entry()
        {
            void *f = nullptr;
            cudaDriverEntryPointQueryResult q;
            if (cudaGetDriverEntryPoint("cuCtxGetCurrent", &f, cudaEnableDefault, &q) ==
                    cudaSuccess && q == cudaDriverEntryPointSuccess)
                current = reinterpret_cast<GetCurrent>(f);
            if (cudaGetDriverEntryPoint("cuCtxGetId", &f, cudaEnableDefault, &q) == cudaSuccess &&
                q == cudaDriverEntryPointSuccess)
                id = reinterpret_cast<GetId>(f);
            (void)cudaGetLastError();
        }
    };
    static const Entry entry;
    if (!entry.current || !entry.id) return 0;
    for (int attempt = 0; attempt < 2; ++attempt) {
        CUcontext c = nullptr;
        unsigned long long id = 0;
        if (entry.current(&c) == CUDA_SUCCESS && c && entry.id(c, &id) == CUDA_SUCCESS) return id;
        // none yet on this thread, or ended by a reset: the runtime's own
        if (attempt == 0 && cudaFree(nullptr) != cudaSuccess) (void)cudaGetLastError();
    }
    return 0;
}

}  // namespace

cudaError_t block_get(Block *b, size_t bytes, bool pinned)
{
    Block n;
    cudaError_t e = cudaGetDevice(&n.device);
    if (e != cudaSuccess) return e;
    n.bytes = bytes;
    n.context = context_id();
    n.pinned = pinned;
    if (n.context != 0) {
        std::lock_guard<std::mutex> lock(g_mu);
        Kept &k = stores()[n.context].kept[pinned];
        // the smallest block that is large enough and not an eighth too large:
        // what a set holds stays what lulesh_footprint_bytes says, nearly
        size_t best = k.blocks.size();
        for (size_t i = 0; i < k.blocks.size(); ++i)
            if (k.blocks[i].bytes >= bytes && k.blocks[i].bytes <= bytes + bytes / 8 + 4096 &&
                (best == k.blocks.size() || k.blocks[i].bytes < k.blocks[best].bytes))
                best = i;
        if (best < k.blocks.size()) {
            *b = k.blocks[best];
            k.bytes -= b->bytes;
            k.blocks.erase(k.blocks.begin() + (long)best);
            return cudaSuccess;
        }
    }
    e = retry_trimmed([&] { return pinned ? cudaMallocHost(&n.p, bytes) : cudaMalloc(&n.p, bytes); });
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
    if (was.context != 0 && context_id() == was.context) {
        std::lock_guard<std::mutex> lock(g_mu);
        Kept &k = stores()[was.context].kept[was.pinned];
        keep = k.blocks.size() < kCacheBlocks &&
               k.bytes + was.bytes <= (was.pinned ? kCachePinnedBytes : kCacheDeviceBytes);
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

bool block_trim()
{
    const unsigned long long context = context_id();
    Store was;
    {
        std::lock_guard<std::mutex> lock(g_mu);
        const auto it = stores().find(context);
        if (it != stores().end()) std::swap(was, it->second);
    }
    for (const Kept &k : was.kept)
        for (const Block &b : k.blocks) free_block(b);
    return !was.kept[0].blocks.empty() || !was.kept[1].blocks.empty();
}

}  // namespace lulesh

extern "C" int lulesh_release_memory(void)
{
    lulesh::block_trim();
    return LULESH_OK;
}
