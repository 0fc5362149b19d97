// mrg8g_batch.cu -- the allocation-free batch entry point
// (mrg8g_batch_generate_noalloc).  The kernels are those of plans (launch_batch).
#include <algorithm>
#include <cstring>
#include <mutex>

#include "../../include/mrg8g.h"
#include "mrg8g_internal.h"
#include "mrg8g_runtime.h"

// Some callers of this library may not allocate device memory themselves:
// plugins whose host application (or a framework's caching allocator) owns
// all of the GPU's memory, and latency-critical loops that cannot afford the
// device-wide synchronisation and unpredictable cost of cudaMalloc/cudaFree.
// For them the batch path runs from a fixed scratch area that lives in this
// module as a file-scope device array: the counter of the work queue, the
// instance descriptors and the tiles.  Every GPU that loads the library holds
// this array (about 1.3 MB) until the process exits.
//
// Layout: [0, 256) work counter | instances (64 B each) | tiles (16 B each).
namespace mrg8g {
namespace {

constexpr size_t kNoAllocInstOff = 256;
constexpr size_t kNoAllocTileOff = kNoAllocInstOff + (size_t)MRG8G_NOALLOC_MAX_INSTANCES * sizeof(BatchInst);
constexpr size_t kNoAllocBytes = kNoAllocTileOff + (size_t)MRG8G_NOALLOC_MAX_TILES * sizeof(BatchTile);
static_assert(sizeof(BatchInst) == 64 && sizeof(BatchTile) == 16, "descriptor layout");
constexpr int kNoAllocTileRows = 512;
constexpr int kMaxDevices = 64;

}  // namespace
}  // namespace mrg8g

static __device__ __align__(256) unsigned char g_noalloc_scratch[mrg8g::kNoAllocBytes];

namespace mrg8g {
namespace {

// Host staging laid out like the device array (one copy per call).
alignas(256) unsigned char g_noalloc_host[kNoAllocBytes];
std::mutex g_noalloc_mu;
void* g_noalloc_dev[kMaxDevices];

// Device address of g_noalloc_scratch on the current device, looked up once
// per device (the host-side name is only a stand-in, never a device address).
int noalloc_scratch(int dev, void** out) {
    if (dev < 0 || dev >= kMaxDevices) return fail(MRG8G_ERR_INVALID_ARGUMENT, "device %d out of range", dev);
    if (!g_noalloc_dev[dev]) {
        void* p = nullptr;
        cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
        if (e != cudaSuccess) return cuda_fail(e, "cudaGetSymbolAddress(no-alloc scratch)");
        g_noalloc_dev[dev] = p;
    }
    *out = g_noalloc_dev[dev];
    return MRG8G_SUCCESS;
}

// Tiles written straight into the staging area (no heap), cut as every plan
// cuts them (mrg8g_tiles.h) and in a plan's order: by kind in a mixed batch, then
// largest first.  Kinds of one order have outputs of one size, so that their full
// tiles come first as they are and only the others (heads and ends) are sorted,
// by an in-place sort: 16 mixed instances of 2^22 outputs 256 microseconds a call
// with all tiles sorted, now 103.
int noalloc_tiles(const BatchInst* insts, uint32_t count, bool mixed, BatchTile* tiles, uint32_t* ntiles) {
    const uint32_t T = (uint32_t)kNoAllocTileRows * 32u * (uint32_t)kBatchLayoutV;
    uint64_t total = 0;
    for (uint32_t i = 0; i < count; ++i) {
        total += instance_tiles(insts[i], T);
        if (total > MRG8G_NOALLOC_MAX_TILES)
            return fail(MRG8G_ERR_BUDGET, "batch needs more than %d tiles (the no-alloc limit)", MRG8G_NOALLOC_MAX_TILES);
    }
    uint32_t k = 0;
    for (int order = 0; order < (mixed ? 3 : 1); ++order) {
        uint32_t parts = 0;
        for (int part = 0; part < 2; ++part) {
            if (part) parts = k;
            for (uint32_t i = 0; i < count; ++i) {
                if (mixed && kind_order(insts[i].kind) != order) continue;
                const uint32_t m = (uint32_t)instance_tiles(insts[i], T);
                // Of m tiles the first may be a head and the last one short.
                for (uint32_t li = 0; li < m; ++li) {
                    if (part && li == 1 && m > 2) li = m - 1;
                    const BatchTile t = derive_tile(li, insts[i], i, T);
                    if ((t.len_flags != T) == (part != 0)) tiles[k++] = t;
                }
            }
        }
        const auto larger = [](const BatchTile& x, const BatchTile& y) {
            const uint32_t nx = x.len_flags & ~kTileHead, ny = y.len_flags & ~kTileHead;
            return nx != ny ? nx > ny : x.inst != y.inst ? x.inst < y.inst : x.start < y.start;
        };
        if (!std::is_sorted(tiles + parts, tiles + k, larger)) std::sort(tiles + parts, tiles + k, larger);
    }
    *ntiles = k;
    return MRG8G_SUCCESS;
}

}  // namespace
}  // namespace mrg8g

extern "C" int mrg8g_batch_generate_noalloc(const mrg8g_instance* inst, uint64_t count, void* stream) {
    using namespace mrg8g;
    if (count && !inst) return fail(MRG8G_ERR_INVALID_ARGUMENT, "null instance array");
    if (count > MRG8G_NOALLOC_MAX_INSTANCES)
        return fail(MRG8G_ERR_BUDGET, "%llu instances exceed the no-alloc limit of %d", (unsigned long long)count,
                    MRG8G_NOALLOC_MAX_INSTANCES);
    // A stream that is capturing would record the descriptor copy below as a
    // graph node reading g_noalloc_host at replay time, after later calls have
    // rewritten it; such calls are refused before anything is enqueued.
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    cudaError_t qe = cudaStreamIsCapturing((cudaStream_t)stream, &cap);
    if (qe != cudaSuccess) {
        cudaGetLastError();
        return cuda_fail(qe, "cudaStreamIsCapturing");
    }
    if (cap != cudaStreamCaptureStatusNone)
        return fail(MRG8G_ERR_INVALID_ARGUMENT, "the no-alloc batch cannot be enqueued on a stream that is capturing");
    int dev = 0;
    int rc = ensure_device(&dev, nullptr);
    if (rc || (rc = check_waits())) return rc;
    std::lock_guard<std::mutex> lk(g_noalloc_mu);
    void* scratch = nullptr;
    if ((rc = noalloc_scratch(dev, &scratch))) return rc;
    BatchInst* h_insts = reinterpret_cast<BatchInst*>(g_noalloc_host + kNoAllocInstOff);
    BatchTile* h_tiles = reinterpret_cast<BatchTile*>(g_noalloc_host + kNoAllocTileOff);
    int kind = -1;
    uint64_t longest = 0;
    for (uint64_t i = 0; i < count; ++i) {
        const mrg8g_instance& s = inst[i];
        kind = i == 0 || kind == s.kind ? s.kind : -1;
        if (!kind_valid(s.kind))
            return fail(MRG8G_ERR_INVALID_ARGUMENT, "instance %llu: unknown kind %d", (unsigned long long)i, s.kind);
        if ((rc = validate_state(s.state))) return rc;
        const int elem = kind_elem_bytes(s.kind);
        if (s.n && (!s.out || (uintptr_t)s.out % elem))
            return fail(MRG8G_ERR_INVALID_ARGUMENT, "instance %llu: null or misaligned output", (unsigned long long)i);
        if (s.n > (1ull << 62) || s.offset > ~0ull - s.n)
            return fail(MRG8G_ERR_INVALID_ARGUMENT, "instance %llu: offset + n overflows", (unsigned long long)i);
        BatchInst& d = h_insts[i];
        std::memcpy(d.st, s.state, sizeof(d.st));
        d.offset = s.offset;
        d.n = s.n;
        d.out = s.out;
        d.kind = s.kind;
        d.slot1 = 0;
        longest = std::max<uint64_t>(longest, s.n);
    }
    uint32_t ntiles = 0;
    if ((rc = noalloc_tiles(h_insts, (uint32_t)count, kind < 0, h_tiles, &ntiles))) return rc;
    if (ntiles == 0) return MRG8G_SUCCESS;
    // The work counter must start at zero; the array keeps the last call's
    // contents, so the copy below rewrites it together with the descriptors.
    std::memset(g_noalloc_host, 0, kNoAllocInstOff);
    cudaStream_t st = (cudaStream_t)stream;
    unsigned char* d = static_cast<unsigned char*>(scratch);
    cudaError_t e;
    if ((e = cudaMemcpyAsync(d, g_noalloc_host, kNoAllocInstOff + count * sizeof(BatchInst), cudaMemcpyHostToDevice,
                             st)) != cudaSuccess ||
        (e = cudaMemcpyAsync(d + kNoAllocTileOff, g_noalloc_host + kNoAllocTileOff, ntiles * sizeof(BatchTile),
                             cudaMemcpyHostToDevice, st)) != cudaSuccess)
        return cuda_fail(e, "copy of the no-alloc descriptors");
    BatchArgs a;
    a.insts = reinterpret_cast<const BatchInst*>(d + kNoAllocInstOff);
    a.tiles = reinterpret_cast<const BatchTile*>(d + kNoAllocTileOff);
    a.ntiles = ntiles;
    a.counter = reinterpret_cast<uint32_t*>(d);
    a.done_blocks = nullptr;
    a.tile_base = nullptr;
    a.ninst = count;
    a.tile_elems = 0;
    a.states = nullptr;
    a.times = nullptr;
    a.fault = device_fault();
    longest = std::min<uint64_t>(longest, (uint64_t)kNoAllocTileRows * 32 * kBatchLayoutV);
    if ((e = launch_batch(a, kind, longest, 128, 0, st)) != cudaSuccess)
        return cuda_fail(e, "launching the no-alloc batch");
    return MRG8G_SUCCESS;
}
