// snn_blocks.cu -- device memory blocks of the handles, and the spare ones.
//
// A handle takes all its buffers from one block (plus one for a loss list and
// one for kept neighbour lists), because every cudaMalloc and cudaFree costs up
// to hundreds of microseconds whatever its size, by machine, and a small selection
// runs for about one millisecond: with a pair per buffer, about 35, whole passes
// over 100 x 10 rows took 2.3 ms on one B200 and 4.8 on another, where a pair costs
// 0.7 ms (now 0.34 and 0.36).  Released small blocks are kept for the next handle, with
// the stream and events of the handle that used them.
//
// Bounds: at most kSpareBlocks blocks and kSpareBytes bytes are kept in the
// process; larger blocks go straight back to CUDA, the oldest spare makes room
// for a newer one, and all of a device's spares are given back when an
// allocation there fails or the program asks (snn_release_memory).  A block is released only after its handle's stream
// has been waited for, so any thread and stream may take it next; the list is
// guarded by a mutex.  A device reset frees blocks behind our back: a spare is
// used only while the driver still knows its allocation by the same buffer id
// (never reused within a process), otherwise it is forgotten.
#include <cuda.h>
#include <cudaTypedefs.h>

#include <mutex>
#include <vector>

#include "snn_internal.h"

namespace snn {

namespace {

constexpr size_t kSpareBytes = (size_t)256 << 20;
constexpr size_t kSpareBlocks = 16;
constexpr size_t kGrain = (size_t)1 << 20;  // block sizes are multiples of it

std::mutex g_mu;
std::vector<Block> g_spare;  // oldest first

PFN_cuPointerGetAttribute_v4000 attribute_fn()
{
    static const PFN_cuPointerGetAttribute_v4000 fn = [] {
        void *p = nullptr;
        cudaDriverEntryPointQueryResult q;
        const bool ok = cudaGetDriverEntryPoint("cuPointerGetAttribute", &p, cudaEnableDefault, &q) == cudaSuccess &&
                        q == cudaDriverEntryPointSuccess;
        if (!ok) cudaGetLastError();
        return reinterpret_cast<PFN_cuPointerGetAttribute_v4000>(ok ? p : nullptr);
    }();
    return fn;
}

// The driver's id of the allocation that holds p; 0 if it has none.
unsigned long long buffer_id(const void *p)
{
    const PFN_cuPointerGetAttribute_v4000 fn = attribute_fn();
    unsigned long long id = 0;
    if (!fn || fn(&id, CU_POINTER_ATTRIBUTE_BUFFER_ID, (CUdeviceptr)(uintptr_t)p) != CUDA_SUCCESS) return 0;
    return id;
}

void destroy(Block &b)
{
    for (EventPair &e : b.events) {
        if (e.a) cudaEventDestroy(e.a);
        if (e.b) cudaEventDestroy(e.b);
    }
    b.events.clear();
    if (b.stream) cudaStreamDestroy(b.stream);
    b.stream = nullptr;
    if (b.base) cudaFree(b.base);
    b.base = nullptr;
}

}  // namespace

cudaError_t block_acquire(int device, size_t bytes, Block *out)
{
    bytes = (bytes + kGrain - 1) / kGrain * kGrain;
    *out = Block();
    if (bytes <= kSpareBytes) {
        std::lock_guard<std::mutex> lk(g_mu);
        for (;;) {  // the smallest that is large enough and not much too large
            size_t best = g_spare.size();
            for (size_t i = 0; i < g_spare.size(); ++i)
                if (g_spare[i].device == device && g_spare[i].bytes >= bytes && g_spare[i].bytes <= 4 * bytes &&
                    (best == g_spare.size() || g_spare[i].bytes < g_spare[best].bytes))
                    best = i;
            if (best == g_spare.size()) break;
            Block b = std::move(g_spare[best]);
            g_spare.erase(g_spare.begin() + best);
            if (buffer_id(b.base) != b.id) continue;  // gone with a device reset, stream and events too
            *out = std::move(b);
            return cudaSuccess;
        }
    }
    void *p = nullptr;
    cudaError_t e = cudaMalloc(&p, bytes);
    if (e == cudaErrorMemoryAllocation) {
        cudaGetLastError();
        blocks_trim(device);
        e = cudaMalloc(&p, bytes);
    }
    if (e != cudaSuccess) {
        cudaGetLastError();
        return e;
    }
    out->device = device;
    out->base = static_cast<char *>(p);
    out->bytes = bytes;
    out->id = bytes <= kSpareBytes ? buffer_id(p) : 0;
    return cudaSuccess;
}

void block_release(Block &b, bool idle)
{
    if (!b.base || !idle || b.id == 0) {
        destroy(b);
        return;
    }
    for (size_t i = b.events.size(); i-- > 0;)  // whole pairs only
        if (!(b.events[i].a && b.events[i].b)) {
            if (b.events[i].a) cudaEventDestroy(b.events[i].a);
            if (b.events[i].b) cudaEventDestroy(b.events[i].b);
            b.events.erase(b.events.begin() + i);
        }
    std::vector<Block> drop;
    {
        std::lock_guard<std::mutex> lk(g_mu);
        size_t sum = b.bytes;
        for (const Block &s : g_spare) sum += s.bytes;
        while (!g_spare.empty() && (sum > kSpareBytes || g_spare.size() >= kSpareBlocks)) {
            sum -= g_spare.front().bytes;
            drop.push_back(std::move(g_spare.front()));
            g_spare.erase(g_spare.begin());
        }
        g_spare.push_back(std::move(b));
    }
    b = Block();
    for (Block &d : drop)
        if (buffer_id(d.base) == d.id) destroy(d);
}

void blocks_trim(int device)
{
    std::vector<Block> drop;
    {
        std::lock_guard<std::mutex> lk(g_mu);
        for (size_t i = g_spare.size(); i-- > 0;)
            if (device < 0 || g_spare[i].device == device) {
                drop.push_back(std::move(g_spare[i]));
                g_spare.erase(g_spare.begin() + i);
            }
    }
    for (Block &d : drop)
        if (buffer_id(d.base) == d.id) destroy(d);
}

}  // namespace snn
