// block_cache.cu -- see block_cache.hpp.
#include "block_cache.hpp"

#include <cuda.h>

#include <map>
#include <mutex>
#include <vector>

#include "lulesh_b200.h"

namespace lulesh {

namespace {

struct Kept {
    std::vector<Block> blocks;
    size_t bytes = 0;
    size_t slack = 0;  // of the blocks in use: what they hold beyond what was asked
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
    n.bytes = n.asked = bytes;
    n.context = context_id();
    n.pinned = pinned;
    if (n.context != 0) {
        std::lock_guard<std::mutex> lock(g_mu);
        Kept &k = stores()[n.context].kept[pinned];
        // the smallest block that is large enough, and that is not an eighth too
        // large, or not twice while the sets in use hold little more than they
        // need: what they hold stays near lulesh_footprint_bytes.  (An eighth
        // alone: 2,000 jobs of any size one after the other at 1.9e9
        // zone-cycles/s on B200, against 2.5e9.)
        const auto fits = [&](const Block &c) {
            if (c.bytes < bytes || c.bytes > 2 * bytes + 4096) return false;
            const size_t over = c.bytes - bytes;
            return over <= bytes / 8 + 4096 || k.slack + over <= kCacheSlackBytes;
        };
        size_t best = k.blocks.size();
        for (size_t i = 0; i < k.blocks.size(); ++i)
            if (fits(k.blocks[i]) &&
                (best == k.blocks.size() || k.blocks[i].bytes < k.blocks[best].bytes))
                best = i;
        if (best < k.blocks.size()) {
            *b = k.blocks[best];
            b->asked = bytes;
            k.bytes -= b->bytes;
            k.slack += b->bytes - bytes;
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
    if (was.context != 0) {
        const bool lives = context_id() == was.context;
        std::lock_guard<std::mutex> lock(g_mu);
        Kept &k = stores()[was.context].kept[was.pinned];
        k.slack -= was.bytes - was.asked;
        keep = lives && k.blocks.size() < kCacheBlocks &&
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
    if (!b->p) return;
    if (b->context != 0) {
        std::lock_guard<std::mutex> lock(g_mu);
        stores()[b->context].kept[b->pinned].slack -= b->bytes - b->asked;
    }
    free_block(*b);
    *b = Block{};
}

bool block_trim()
{
    const unsigned long long context = context_id();
    std::vector<Block> was;
    {
        std::lock_guard<std::mutex> lock(g_mu);
        const auto it = stores().find(context);
        if (it == stores().end()) return false;
        for (Kept &k : it->second.kept) {
            was.insert(was.end(), k.blocks.begin(), k.blocks.end());
            k.blocks.clear();
            k.bytes = 0;
        }
    }
    for (const Block &b : was) free_block(b);
    return !was.empty();
}

}  // namespace lulesh

extern "C" int lulesh_release_memory(void)
{
    lulesh::block_trim();
    return LULESH_OK;
}
