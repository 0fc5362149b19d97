// mrg8g_plain.cu -- the recurrence kernels for sm_103a (small single-stream calls
// and batches) and their small companions (device jump of many offsets, integer ->
// uniform conversion).
//
// Replaces rng_outer_32 / rng_inner of cuda/mrg8_cuda.cu:201-399.  Layout of
// the work: the call's n outputs (stream positions 0..n-1 after the handle's
// current state) are cut into one contiguous tile per warp.  A warp jumps its
// state to the tile start with the resident byte-window jump table, then lane l owns V
// interleaved decimated substreams (positions B + V l + v + 32 V j); each is
// an order-8 recurrence of its own (coefficients of the characteristic
// polynomial of A^(32V)), so a lane needs 8 multiply-adds per output, no
// shuffles and no shared memory after its setup, and every row j of the warp is one
// contiguous 32 V-element run written with 16-byte vector stores.
#include "mrg8g_device.cuh"
#include "mrg8g_gen.cuh"
#include "mrg8g_internal.h"
#include "mrg8g_runtime.h"

namespace mrg8g {

MRG8G_DEFINE_TABLE_UPLOAD(upload_tables_plain)

// Resident blocks the register allocation must allow: eight for 4-byte
// outputs with four substreams per lane (64 registers); nine for fp64
// ORIGINAL with two (56 registers instead of 64: 718 against 710
// Goutputs/s); else no bound (fp64 SHIFTED measured 791 Goutputs/s
// unbounded, 56 registers, and 772 when held to 48 for ten blocks per SM).
template <int V, int KIND>
constexpr int plain_min_blocks() {
    return (V == 4 && sizeof(typename OutOf<KIND>::T) == 4) ? 8 : (V == 2 && KIND == kF64Orig) ? 9 : 1;
}

template <int V, int KIND>
__global__ void __launch_bounds__(kPlainThreads, plain_min_blocks<V, KIND>())
    k_plain(const __grid_constant__ PlainArgs a) {
    using T = typename OutOf<KIND>::T;
    __shared__ __align__(16) uint32_t scratch[kPlainThreads / 32][window_scratch(V)];
    T* const out = static_cast<T*>(a.out);
    const int lane = threadIdx.x & 31;
    const uint64_t warp = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;

    // Unaligned head: the first `head` (< V) outputs, one lane, sequential.
    if (warp == 0 && lane == 0 && a.head) {
        after_previous_kernel();
        uint32_t st[8];
#pragma unroll
        for (int q = 0; q < 8; ++q) st[q] = a.st[q];
        lane_sequential<KIND>(g_jwin, st, out, a.head);  // row 0 of A = coefficients
    }

    const uint64_t B = a.head + warp * a.tile;
    if (B >= a.n) return;
    uint32_t s[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) s[q] = a.st[q];
    warp_jump(g_jwin, s, B);
    after_previous_kernel();
    // Not sooner: the next kernel's blocks may take what the kernel before still needs.
    if (threadIdx.x == 0) next_kernel_may_start();
    warp_generate<V, KIND>(g_win, g_dstep, s, out + B, min(a.tile, a.n - B), a.lc, scratch[threadIdx.x >> 5]);
}

// ---- batches (BatchArgs): one tile per warp at a time.  Small batches, whose time
// is their latency, and launches of few resident blocks (recurrence_blocks
// in mrg8g_tiles.h); the others run k_tensor_batch.

// The batch layout's recurrence: [0] lags S - 1, [1] lags S mod p.  An argument:
// from constant memory its first use cost a launch about half a microsecond.
struct BatchLeaps {
    LeapCoef lc[2];
};

// Tiles shorter than this many outputs (256 rows) form their windows in one table
// round trip even in a launch with more tiles than warps: there the setup is a
// large part of the tile (65,536 tiles of 4,096 outputs: 818 against 754 Goutputs/s).
constexpr uint32_t kQuickSetupElems = 256u * 32u * kBatchLayoutV;

template <int KIND, bool QUICK>
__device__ __forceinline__ void run_tile(const BatchInst& in, const BatchTile& t, const uint32_t s[8],
                                         const BatchLeaps& leaps, uint32_t* scratch) {
    using T = typename OutOf<KIND>::T;
    warp_generate<kBatchLayoutV, KIND>(g_win, g_dstep, s, static_cast<T*>(in.out) + t.start, t.len_flags,
                                       leaps.lc[kLagMod<KIND> ? 1 : 0], scratch,
                                       QUICK || t.len_flags < kQuickSetupElems);
}

// Instance owning tile ti of a device-tiled launch: the largest i with
// tile_base[i] <= ti, found by a 32-way search (one load per lane per level,
// one level for up to 32 instances).  Called by all 32 lanes with the same ti.
__device__ __forceinline__ uint32_t tile_owner(const uint32_t* __restrict__ base, uint32_t ninst, uint32_t ti) {
    const int lane = threadIdx.x & 31;
    uint32_t lo = 0, hi = ninst;  // base[lo] <= ti < base[hi]
    while (hi - lo > 1) {
        const uint32_t step = (hi - lo + 31) / 32;
        const uint32_t c = lo + (uint32_t)lane * step;
        const unsigned m = __ballot_sync(kFull, c < hi && base[c] <= ti);
        lo += (uint32_t)(31 - __clz((int)m)) * step;
        hi = min(hi, lo + step);
    }
    return lo;
}

// QUICK: a launch with no more tiles than warps: each warp takes the tile of its
// own index in the grid (no wait on the counter) and forms its window in one table
// round trip.  Otherwise warps pull tiles from the counter.
template <int THREADS, bool QUICK>
__global__ void __launch_bounds__(THREADS, THREADS == 128 ? 9 : 4) k_batch(const __grid_constant__ BatchArgs a,
                                                                                const __grid_constant__ BatchLeaps leaps) {
    if (a.times && blockIdx.x == 0 && threadIdx.x == 0) a.times[0] = global_ns();
    __shared__ __align__(16) uint32_t scratch[THREADS / 32][window_scratch(kBatchLayoutV)];
    const int lane = threadIdx.x & 31;
    uint32_t* sc = scratch[threadIdx.x >> 5];
    for (int round = 0;; ++round) {
        uint32_t ti;
        if constexpr (QUICK) {
            if (round) break;
            ti = blockIdx.x * (THREADS / 32) + (threadIdx.x >> 5);
        } else {
            uint32_t q = 0;
            if (lane == 0) q = atomicAdd(a.counter, 1u);
            ti = __shfl_sync(kFull, q, 0);
        }
        if (ti >= a.ntiles) break;
        BatchTile t;
        BatchInst in;
        if (a.tiles) {
            t = a.tiles[ti];
            in = a.insts[t.inst];
        } else {
            const uint32_t i = tile_owner(a.tile_base, a.ninst, ti);
            in = a.insts[i];
            t = derive_tile(ti - a.tile_base[i], in, i, a.tile_elems);
        }
        const uint32_t* src = in.slot1 ? a.states + 8ull * (in.slot1 - 1) : in.st;
        uint32_t s[8];
#pragma unroll
        for (int q = 0; q < 8; ++q) s[q] = src[q];
        warp_jump(g_jwin, s, in.offset + t.start);
        if (t.len_flags & kTileHead) {
            if (lane == 0)
                write_head(g_jwin, in.kind, s, (char*)in.out + t.start * tile_elem_bytes(in.kind), t.len_flags & ~kTileHead);
            continue;
        }
        switch (in.kind) {
        case kU32: run_tile<kU32, QUICK>(in, t, s, leaps, sc); break;
        case kF64Orig: run_tile<kF64Orig, QUICK>(in, t, s, leaps, sc); break;
        case kF64Shift: run_tile<kF64Shift, QUICK>(in, t, s, leaps, sc); break;
        case kF32Orig: run_tile<kF32Orig, QUICK>(in, t, s, leaps, sc); break;
        default: run_tile<kF32Shift, QUICK>(in, t, s, leaps, sc); break;
        }
    }
    leave_queue(a);
}

// Uniforms from raw stream integers S in [1, p] (grid-stride).
template <int KIND>
__global__ void k_convert(const uint32_t* __restrict__ in, typename OutOf<KIND>::T* __restrict__ out,
                          uint64_t n) {
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
         i += (uint64_t)gridDim.x * blockDim.x)
        out[i] = convert<KIND>(lag_of<KIND>(in[i]));
}

// states[8 i .. 8 i + 7] = A^offsets[i] st, eight lanes per offset.  Offsets
// below 8 step sequentially (raw words shift through unchanged, as in the
// reference); larger ones jump and come back as representatives in [1, p].
// Bound by the traffic and the latency of the table's rows (2 KB per jump from
// L1 and L2) beside the products.  GB300, offsets below 2^63, against one warp
// per offset (warp_jump): 65,536 offsets 37.0 -> 16.6 microseconds, 2^20 of them
// 524 -> 196, 100 alike (4.5).  Rows two byte positions at a time 20.7, eight at
// a time 26.7, 32-byte loads 22.6, signed entries with one sum 20.7, the words
// exchanged through shared memory no different.
__global__ void __launch_bounds__(kPlainThreads)
    k_jump_states(const __grid_constant__ JumpArgs a) {
    const int lane = threadIdx.x & 31, r = lane & 7;
    const uint64_t nwarps = ((uint64_t)gridDim.x * blockDim.x) >> 5;
    for (uint64_t w = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; 4 * w < a.count; w += nwarps) {
        const uint64_t i = 4 * w + (lane >> 3);
        const uint64_t k = i < a.count ? a.offsets[i] : 0;
        uint32_t s[8];
#pragma unroll
        for (int q = 0; q < 8; ++q) s[q] = a.st[q];
        group_jump(g_jwin, s, k < 8 ? 0 : k);
        if (k < 8) {
            for (uint64_t n = 0; n < k; ++n) {
                const uint32_t S = dot8_ref(g_jwin, s);  // row 0 of A
#pragma unroll
                for (int q = 7; q > 0; --q) s[q] = s[q - 1];
                s[0] = S;
            }
        } else {
#pragma unroll
            for (int q = 0; q < 8; ++q) s[q] = rep1p(s[q]);
        }
        uint32_t mine = s[0];
#pragma unroll
        for (int q = 1; q < 8; ++q) mine = r == q ? s[q] : mine;
        if (i < a.count) a.states[i * 8 + r] = mine;
    }
}

// ------------------------------------------------------------- launchers

template <int V, int KIND>
static cudaError_t launch_plain_t(const PlainArgs& a, int blocks, cudaStream_t st) {
    // A call of one block may overlap the kernel before it.  Larger ones must not:
    // their blocks would pile up on the SMs that come free first (2^22 uint32 with
    // four substreams per lane: 12 -> 27 microseconds).
    if (blocks == 1) return launch_overlapped(k_plain<V, KIND>, blocks, kPlainThreads, 0, st, a);
    k_plain<V, KIND><<<blocks, kPlainThreads, 0, st>>>(a);
    return cudaGetLastError();
}

template <int V, int KIND>
static int occupancy_t() {
    int nb = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, k_plain<V, KIND>, kPlainThreads, 0) != cudaSuccess)
        return 1;
    return nb > 0 ? nb : 1;
}

#define MRG8G_KIND_SWITCH(V, FN, ...)                       \
    switch (kind) {                                         \
    case kU32: return FN<V, kU32>(__VA_ARGS__);             \
    case kF64Orig: return FN<V, kF64Orig>(__VA_ARGS__);     \
    case kF64Shift: return FN<V, kF64Shift>(__VA_ARGS__);   \
    case kF32Orig: return FN<V, kF32Orig>(__VA_ARGS__);     \
    default: return FN<V, kF32Shift>(__VA_ARGS__);          \
    }

cudaError_t launch_plain(int kind, int V, const PlainArgs& a, int blocks, cudaStream_t st) {
    if (V == 1) { MRG8G_KIND_SWITCH(1, launch_plain_t, a, blocks, st) }
    if (V == 2) { MRG8G_KIND_SWITCH(2, launch_plain_t, a, blocks, st) }
    MRG8G_KIND_SWITCH(4, launch_plain_t, a, blocks, st)
}

int plain_blocks_per_sm(int kind, int V) {
    if (V == 1) { MRG8G_KIND_SWITCH(1, occupancy_t) }
    if (V == 2) { MRG8G_KIND_SWITCH(2, occupancy_t) }
    MRG8G_KIND_SWITCH(4, occupancy_t)
}

cudaError_t launch_batch_recurrence(const BatchArgs& a, int threads, int blocks, cudaStream_t st) {
    const HostTables& t = host_tables();
    const BatchLeaps leaps = {{t.leap[layout_index(kBatchLayoutV)], t.leap_mod[layout_index(kBatchLayoutV)]}};
    const bool quick = (uint64_t)a.ntiles <= (uint64_t)blocks * (uint64_t)(threads / 32);
    if (threads == 256) {
        if (quick) k_batch<256, true><<<blocks, 256, 0, st>>>(a, leaps);
        else k_batch<256, false><<<blocks, 256, 0, st>>>(a, leaps);
    } else {
        if (quick) k_batch<128, true><<<blocks, 128, 0, st>>>(a, leaps);
        else k_batch<128, false><<<blocks, 128, 0, st>>>(a, leaps);
    }
    return cudaGetLastError();
}

int batch_blocks_per_sm(int threads) {
    int nb = 0;
    const cudaError_t e = threads == 256
                              ? cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, k_batch<256, false>, 256, 0)
                              : cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, k_batch<128, false>, 128, 0);
    return e == cudaSuccess && nb > 0 ? nb : 1;
}

cudaError_t launch_convert(int kind, const uint32_t* in, void* out, uint64_t n, int blocks, cudaStream_t st) {
    switch (kind) {
    case kF64Orig: k_convert<kF64Orig><<<blocks, 256, 0, st>>>(in, (uint64_t*)out, n); break;
    case kF64Shift: k_convert<kF64Shift><<<blocks, 256, 0, st>>>(in, (uint64_t*)out, n); break;
    case kF32Orig: k_convert<kF32Orig><<<blocks, 256, 0, st>>>(in, (uint32_t*)out, n); break;
    case kF32Shift: k_convert<kF32Shift><<<blocks, 256, 0, st>>>(in, (uint32_t*)out, n); break;
    default: return cudaErrorInvalidValue;
    }
    return cudaGetLastError();
}

cudaError_t launch_jump_states(const JumpArgs& a, int blocks, cudaStream_t st) {
    k_jump_states<<<blocks, kPlainThreads, 0, st>>>(a);
    return cudaGetLastError();
}

}  // namespace mrg8g
