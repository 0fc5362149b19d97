// mrg8g_tensor.cu -- generation on the tensor cores (tcgen05).
//
// A block of 256 outputs is a constant matrix times its start state
// (TensorTables in mrg8g_tables.h): with the state's 32 bytes as fp16 and the
// coefficients as three signed 11-bit limbs, one step of 32 blocks is three
// 128 x 64 x 48 products whose fp32 sums are exact integers, and an output
// takes two wide multiply-adds and two integer operations to put together, where
// the recurrence of mrg8g_gen.cuh takes nine multiply-adds and four.
//
// One block of threads per SM:
//   producers   3 warps.  Each owns a run of steps, lane l holding the start
//               state of block l of the next step; it writes the states'
//               bytes as the fp16 operand of that step and moves the states
//               one step on (64 multiply-adds per 256 outputs).
//   issuer      one lane.  Issues the 9 products of each step, in the order in
//               which the producers finished them, into one of two tensor
//               memory buffers.
//   writers     16 warps, 8 per buffer.  Warp w reads tensor memory lanes
//               32 (w % 4) .. + 31 of half of the step's blocks, finishes the
//               outputs and stores them, 512 (fp64) or 256 bytes per store
//               instruction and 512 consecutive outputs per quarter.
// What bounds it: fp64 the writes (7.2 to 7.4 TB/s at 2^30 outputs by the GPU, against
// 6.7 for a copy and 7.7 for memset), 4-byte kinds the integer pipes and the writes
// (uint32 7.05 TB/s, fp32 5.55).  GB300, 2^30 outputs, this kernel against k_plain:
// uint32 1,763 / 1,040 Goutputs/s, fp32 1,387 / 870, fp64 SHIFTED 900 / 793, ORIGINAL
// 915 / 756; 2^24 fp64 22.5 / 33 microseconds.  Measured on the way, uint32 /
// fp32 / fp64: six matrices of 32 columns (the second outputs of a pair from
// rows of their own) 1,157 / 927 / 802, the products then bound by reading the
// matrices from shared memory; both accumulators shared by all writers 1,500 /
// 1,067 / 873; loads of a chunk only after the one before is stored 1,495 / 1,130
// / 923; a warp's outputs 64 at a time instead of 512 consecutive ones 1,742 /
// 1,347 / 876; two blocks of threads per SM with one accumulator each 1,427 /
// 1,056 / 885.
// The waits for copies, products and other warps are on shared-memory barriers and
// bounded (kWaitLimitNs): one that gives up ends its block, once the block's copies and
// products have ended, and sets the word *fault in host memory.  Two waits are the
// hardware's and end with other kernels: for the kernel before on the stream
// (after_previous_kernel) and for tensor memory that a kernel of another stream
// holds on the SM (tmem_alloc).
#include "mrg8g_device.cuh"
#include "mrg8g_internal.h"
#include "mrg8g_gen.cuh"
#include "mrg8g_tc.cuh"
#include "mrg8g_tiles.h"

namespace mrg8g {

static __device__ __align__(16) uint32_t g_jwin[kJumpWinMats * 64];
static __device__ __align__(128) uint16_t g_tc_a[kTcMats * kTcMatHalves];
static __device__ __align__(128) uint32_t g_tc_col[16 * 32 * 4];
// Constant memory, not an argument: a launch with 0.4 KB more of arguments took
// the host about 1 microsecond longer.
static __constant__ StepCoef c_step, c_quarter;

cudaError_t upload_tables_tensor() {
    const HostTables& t = host_tables();
    cudaError_t e = cudaMemcpyToSymbol(g_jwin, t.jwin, sizeof(g_jwin));
    if (e != cudaSuccess) return e;
    e = cudaMemcpyToSymbol(g_tc_a, t.tc.a, sizeof(g_tc_a));
    if (e != cudaSuccess) return e;
    e = cudaMemcpyToSymbol(g_tc_col, t.tc.col, sizeof(g_tc_col));
    if (e != cudaSuccess) return e;
    e = cudaMemcpyToSymbol(c_step, &t.tc.step, sizeof(c_step));
    if (e != cudaSuccess) return e;
    return cudaMemcpyToSymbol(c_quarter, &t.tc.quarter, sizeof(c_quarter));
}

namespace {

constexpr int kAccs = 2;                  // accumulator buffers in tensor memory, each with writers of its own
constexpr int kWriters = 16;
constexpr int threads_for(int producers) { return 32 * (kWriters + producers + 1); }
constexpr int kRing = 32;                 // step descriptors (more than the operand buffers, accumulators and the end)
constexpr int kAccCols = kTcMats * kTcN;
constexpr int kTmemCols = 512;
constexpr uint32_t kEndKind = 0xFFu;
constexpr int kMixed = -1;

// A quarter of a step as its writers see it: eight blocks of one stream.
struct __align__(16) Quarter {
    unsigned long long out;  // address of its first output
    uint32_t count;          // outputs to write, at most kTcQuarter
    uint32_t kind;
};

template <int PRODUCERS>
struct __align__(128) Shared {
    static constexpr int kProducers = PRODUCERS, kSlots = 2 * PRODUCERS;  // two operand buffers per producer
    static constexpr int kThreads = threads_for(PRODUCERS);
    static_assert(kSlots + kAccs + 2 <= kRing, "ring of step descriptors");
    uint16_t a[kTcMats * kTcMatHalves];
    uint32_t col[16 * 32 * 4];
    uint16_t b[kSlots][kTcN * kTcK];
    Quarter ring[kRing][4];
    uint32_t ring_slot[kRing];
    unsigned long long bar_tables, bar_ready[kRing], bar_free[kSlots], bar_full[kAccs], bar_empty[kAccs];
    uint32_t tmem, next, ended, gave_up;
};

// Where all warps of a bulk launch's block meet, each once and converged: the
// kernel before has completed and the block owns its tensor memory.
template <class Sh>
__device__ __forceinline__ void meet() {
    asm volatile("bar.sync 1, %0;" ::"n"(Sh::kThreads) : "memory");
}

// Two bytes of w (positions in SEL) as fp16 values less 128: 0x6400 + b is
// 1024 + b.
template <uint32_t SEL>
__device__ __forceinline__ uint32_t bytes_as_half2(uint32_t w) {
    const uint32_t h = __byte_perm(w, 0x64646464u, SEL);
    uint32_t r;
    asm("sub.rn.f16x2 %0, %1, %2;" : "=r"(r) : "r"(h), "r"(0x64806480u));  // 1152, 1152
    return r;
}

// Operand row `row` of a slot from the bytes of eight words (h: bytes_as_half2
// of each), and its constants (takes_s: kTakesS of the kind).
__device__ __forceinline__ void write_row(uint16_t* b, const uint2 (&h)[8], int row, bool takes_s) {
#pragma unroll
    for (int c = 0; c < 4; ++c)
        *reinterpret_cast<uint4*>(b + tc_half(row, 8 * c, kTcN / 8)) =
            make_uint4(h[2 * c].x, h[2 * c].y, h[2 * c + 1].x, h[2 * c + 1].y);
    *reinterpret_cast<uint4*>(b + tc_half(row, 32, kTcN / 8)) =
        make_uint4(0x3C006C00u, takes_s ? 0x00003C00u : 0u, 0u, 0u);  // 4096, 1, takes_s
}

__device__ __forceinline__ uint2 word_as_halves(uint32_t w) {
    return make_uint2(bytes_as_half2<0x4140>(w), bytes_as_half2<0x4342>(w));
}

// The lane's two rows: its state, and the state one output later.
__device__ __forceinline__ void write_operand(uint16_t* b, const StepCoef& step, const uint32_t (&s)[8], int lane,
                                              bool takes_s) {
    uint2 h[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) h[q] = word_as_halves(s[q]);
    write_row(b, h, lane, takes_s);
    uint64_t acc = step.K1;
#pragma unroll
    for (int q = 0; q < 8; ++q) acc = mad_wide_s32(step.c1[q], s[q], acc);
#pragma unroll
    for (int q = 7; q > 0; --q) h[q] = h[q - 1];
    h[0] = word_as_halves(reduce_acc(acc));
    write_row(b, h, kTcCols + lane, takes_s);
}

template <int KIND>
constexpr int kElemBytes = KIND == kF64Orig || KIND == kF64Shift ? 8 : 4;

// The ORIGINAL scalings and the integers take the stream value S in [1, p],
// the SHIFTED ones S - 1.
template <int KIND>
constexpr bool kTakesS = KIND == kU32 || KIND == kF64Orig || KIND == kF32Orig;

// One output's S or S - 1 from its three words (TensorTables): y in [1, 2 p)
// is negative as a signed word above p, where y - p is positive.
template <int KIND>
__device__ __forceinline__ uint32_t join(uint32_t w0, uint32_t w1, uint32_t w2) {
    const uint64_t v = (uint64_t)w2 * (1u << 22) + (uint64_t)w1 * (1u << 11);  // < 2^53
    const uint32_t y = ((uint32_t)v >> 1) + (uint32_t)(v >> 32) + w0;
    const uint32_t z = y - kP;
    if constexpr (kTakesS<KIND>) return (uint32_t)max((int)y, (int)z);
    else return min(y, z);
}

// Whether any v of the words put together so far was one of the few that
// f64_bits_fma and f32_bits_fma (mrg8g_arith.cuh) leave out: about one in
// 4 million and one in a million.
template <int KIND>
struct Few {
    uint32_t low = 0xFFFFFFFFu;  // fp64: smallest xn + 512 mod 2^32
    float far = 0.0f;            // fp32: largest |fh - 1/2|
    __device__ __forceinline__ bool any() const {
        if constexpr (KIND == kU32) return false;
        else if constexpr (sizeof(typename OutOf<KIND>::T) == 8) return low <= 512u;
        else return f32_fma_rare(far);
    }
};

// Two outputs' words: the rounding is on the FP32 pipes, since the integer ALU
// bounds the writers (fp32 at 2^30 with the conversion of mrg8g_gen.cuh: 1,085
// against 1,370 Goutputs/s).
template <int KIND>
__device__ __forceinline__ void words_of(uint32_t va, uint32_t vb, typename OutOf<KIND>::T& a,
                                         typename OutOf<KIND>::T& b, Few<KIND>& few) {
    if constexpr (KIND == kU32) {
        a = va;
        b = vb;
    } else if constexpr (sizeof(typename OutOf<KIND>::T) == 8) {
        uint32_t xa, xb;
        a = f64_bits_fma(va, xa);
        b = f64_bits_fma(vb, xb);
        few.low = __vimin3_u32(few.low, xa + 512u, xb + 512u);
    } else {
        float fa, fb;
        a = f32_bits_fma(va, fa);
        b = f32_bits_fma(vb, fb);
        few.far = fmaxf(fmaxf(few.far, fabsf(__fsub_rn(fa, 0.5f))), fabsf(__fsub_rn(fb, 0.5f)));
    }
}

// The word of any v.
template <int KIND>
__device__ __forceinline__ typename OutOf<KIND>::T any_word_of(uint32_t v) {
    if constexpr (KIND == kU32) return v;
    else if constexpr (sizeof(typename OutOf<KIND>::T) == 8) return f64_bits_to_p(v);
    else return f32_bits_fp(v);
}

// Words of kChunk blocks: w[3 i + j] for matrix j and the blocks' rows i.
constexpr int kChunk = 4;
using Words = uint32_t[2 * kTcMats][kChunk];

// The lane's two outputs of kChunk blocks.  p: the first of them; left: outputs
// from there to the quarter's end, looked at if not FULL; plus: added to the
// joined value (0, or 1 to make S of S - 1 in a mixed batch).
template <int KIND, bool FULL>
__device__ __forceinline__ void write_blocks(const Words& w, typename OutOf<KIND>::T* p, int left, uint32_t plus) {
    using T = typename OutOf<KIND>::T;
    if (!FULL && left <= 0) return;
    Few<KIND> few;
#pragma unroll
    for (int c = 0; c < kChunk; ++c) {
        T a, b;
        words_of<KIND>(join<KIND>(w[0][c], w[1][c], w[2][c]) + plus, join<KIND>(w[3][c], w[4][c], w[5][c]) + plus, a, b,
                       few);
        T* const q = p + c * 64;
        if (FULL) {
            if constexpr (sizeof(T) == 8) *reinterpret_cast<ulonglong2*>(q) = make_ulonglong2(a, b);
            else *reinterpret_cast<uint2*>(q) = make_uint2(a, b);
        } else {
            if (c * 64 < left) q[0] = a;
            if (c * 64 + 1 < left) q[1] = b;
        }
    }
    if (few.any()) {  // all of them again, the general way
#pragma unroll
        for (int i = 0; i < 2 * kChunk; ++i) {
            const uint32_t v = join<KIND>(w[3 * (i & 1)][i >> 1], w[3 * (i & 1) + 1][i >> 1], w[3 * (i & 1) + 2][i >> 1]);
            const int o = (i >> 1) * 64 + (i & 1);
            if (FULL || o < left) p[o] = any_word_of<KIND>(v + plus);
        }
    }
}

// Chunk c of quarter q.
template <int KIND>
__device__ __forceinline__ void write_chunk(const Words& w, const Quarter& q, int at, int c, uint32_t plus = 0) {
    typename OutOf<KIND>::T* const p = (typename OutOf<KIND>::T*)q.out + at;
    if (q.count == kTcQuarter) write_blocks<KIND, true>(w, p + c * kChunk * 64, 0, plus);
    else write_blocks<KIND, false>(w, p + c * kChunk * 64, (int)q.count - at - c * kChunk * 64, plus);
}

// KIND: the launch's kind, or kMixed: the code of three kinds then, the
// ORIGINAL scalings as SHIFTED ones of S, because the instruction cache is what
// the writers of a mixed batch wait for.
template <int KIND>
__device__ __forceinline__ void write_any(const Words& w, const Quarter& q, int at, int c) {
    if constexpr (KIND != kMixed) write_chunk<KIND>(w, q, at, c);
    else if (q.kind == kU32) write_chunk<kU32>(w, q, at, c);
    else if (q.kind == kF64Orig || q.kind == kF64Shift) write_chunk<kF64Shift>(w, q, at, c, q.kind == kF64Orig);
    else write_chunk<kF32Shift>(w, q, at, c, q.kind == kF32Orig);
}
// Whether the products are to give S rather than S - 1.
template <int KIND>
__device__ __forceinline__ bool takes_s(uint32_t kind) {
    if constexpr (KIND != kMixed) return kTakesS<KIND>;
    else return kind == kU32;
}

__device__ __forceinline__ void load_words(Words& w, uint32_t addr) {
#pragma unroll
    for (int j = 0; j < 2 * kTcMats; ++j) tmem_ld(w[j], addr + (j % kTcMats) * kTcN + (j / kTcMats) * kTcCols);
}

// A warp writes two quarters of every step of its accumulator, in four chunks,
// each read from tensor memory while the one before is finished and stored.
template <int KIND, class Sh>
__device__ __forceinline__ void writer(Sh& sh, int warp, int lane) {
    const uint32_t acc = warp >> 3, part = (warp >> 2) & 1;
    const uint32_t empty = smem_addr(&sh.bar_empty[acc]), full = smem_addr(&sh.bar_full[acc]);
    const int at = tc_row(32 * (warp & 3) + lane);
    // Tensor memory lane 32 (warp % 4), in bits 16..31.
    const uint32_t addr = sh.tmem + ((uint32_t)(warp & 3) << 21) + acc * kAccCols + part * 16;
    uint32_t phase = 0;
    for (uint32_t t = acc;; t += kAccs, phase ^= 1) {
        if (!__all_sync(kFull, mbar_wait(full, phase, &sh.gave_up))) return;
        tc_fence_after();
        Words w[2];
        load_words(w[0], addr);
        const Quarter q0 = sh.ring[t % kRing][2 * part], q1 = sh.ring[t % kRing][2 * part + 1];
        if (q0.kind == kEndKind) {
            tmem_wait_ld();
            return;
        }
        const auto quarter = [&](const Quarter& q, int i) {
            tmem_wait_ld();
            load_words(w[1], addr + 8 * i + 4);
            write_any<KIND>(w[0], q, at, 0);
            tmem_wait_ld();
            if (i == 0) {
                load_words(w[0], addr + 8);
            } else {  // all read: the accumulator is free for the next products
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(empty);
            }
            write_any<KIND>(w[1], q, at, 1);
        };
        // Rolled for mixed batches (instruction cache); the two other forms differ
        // in what the compiler makes of them (2^30 outputs, straight / unrolled:
        // fp32 781 / 794 microseconds, fp64 1,187 / 1,171).
        if constexpr (KIND != kMixed && kElemBytes<KIND> == 4) {
            quarter(q0, 0);
            quarter(q1, 1);
        } else {
#pragma unroll(KIND == kMixed ? 1 : 2)
            for (int i = 0; i < 2; ++i) {
                Quarter q;  // field by field, to stay in registers
                q.out = i ? q1.out : q0.out;
                q.count = i ? q1.count : q0.count;
                q.kind = i ? q1.kind : q0.kind;
                quarter(q, i);
            }
        }
    }
}

template <class Sh>
__device__ __forceinline__ void issuer(Sh& sh) {
    if (!mbar_wait(smem_addr(&sh.bar_tables), 0, &sh.gave_up)) return;
    const uint32_t a0 = smem_addr(sh.a);
    for (uint32_t t = 0;; ++t) {
        const uint32_t acc = t % kAccs, full = smem_addr(&sh.bar_full[acc]);
        if (!mbar_wait(smem_addr(&sh.bar_ready[t % kRing]), (t / kRing) & 1, &sh.gave_up)) return;
        if (!mbar_wait(smem_addr(&sh.bar_empty[acc]), ((t / kAccs) & 1) ^ 1, &sh.gave_up)) return;
        tc_fence_after();
        if (sh.ring[t % kRing][0].kind == kEndKind) {  // no products: each barrier's two arrivals
            for (uint32_t i = t; i < t + kAccs; ++i) {
                if (!mbar_wait(smem_addr(&sh.bar_empty[i % kAccs]), ((i / kAccs) & 1) ^ 1, &sh.gave_up)) return;
                mbar_arrive(smem_addr(&sh.bar_full[i % kAccs]));
                mbar_arrive(smem_addr(&sh.bar_full[i % kAccs]));
            }
            return;
        }
        const uint32_t slot = sh.ring_slot[t % kRing], b0 = smem_addr(sh.b[slot]);
#pragma unroll
        for (int i = 0; i < kTcMats; ++i)
#pragma unroll
            for (int k = 0; k < kTcK / 16; ++k)
                tc_mma_f16(sh.tmem + acc * kAccCols + i * kTcN,
                           tc_operand(a0 + (i * kTcMatHalves + k * 2 * kTcM * 8) * 2, kTcM * 16, 128),
                           tc_operand(b0 + k * 2 * kTcN * 16, kTcN * 16, 128), tc_f16_desc(kTcN), k > 0);
        tc_commit(smem_addr(&sh.bar_free[slot]));
        tc_commit(full);
        mbar_arrive(full);  // orders the descriptor for the writers
    }
}

// The lane's state is multiplied by the constant matrix of `step`.
__device__ __forceinline__ void advance(uint32_t (&s)[8], const StepCoef& step) {
    uint32_t z[8];
#pragma unroll
    for (int r = 0; r < 8; ++r) {
        uint64_t acc = step.K[r];
#pragma unroll
        for (int q = 0; q < 8; ++q) acc = mad_wide_s32(step.c[r * 8 + q], s[q], acc);
        z[r] = reduce_acc(acc);
    }
#pragma unroll
    for (int r = 0; r < 8; ++r) s[r] = z[r];
}

// The tables in shared memory are there; false if the wait gave up.  Producers
// jump first: the copies arrive meanwhile.
template <class Sh>
__device__ __forceinline__ bool tables_ready(Sh& sh) {
    return __all_sync(kFull, mbar_wait(smem_addr(&sh.bar_tables), 0, &sh.gave_up));
}

// The state at the start of block l of a step that begins at s.
template <class Sh>
__device__ __forceinline__ void to_block(const Sh& sh, uint32_t (&s)[8], int l) {
    uint32_t z[8];
    const uint4* col = reinterpret_cast<const uint4*>(sh.col) + l;
#pragma unroll
    for (int r = 0; r < 8; ++r) {
        const uint4 c0 = col[(2 * r) * 32], c1 = col[(2 * r + 1) * 32];
        const uint32_t m[8] = {c0.x, c0.y, c0.z, c0.w, c1.x, c1.y, c1.z, c1.w};
        z[r] = dot8_ref(m, s);
    }
#pragma unroll
    for (int r = 0; r < 8; ++r) s[r] = z[r];
}

__device__ __forceinline__ uint32_t elem_bytes(int kind) { return kind == kF64Orig || kind == kF64Shift ? 8u : 4u; }

// One step: the lane's block starts at s; lanes 0, 8, 16 and 24 hold the
// step's quarters.  `used`: steps of this producer so far.
template <int KIND, class Sh>
__device__ __forceinline__ bool produce_step(Sh& sh, int producer, int lane, uint32_t& used,
                                             const uint32_t (&s)[8], const Quarter& q) {
    const uint32_t slot = producer * 2 + (used & 1);
    if (!__all_sync(kFull, mbar_wait(smem_addr(&sh.bar_free[slot]), ((used >> 1) & 1) ^ 1, &sh.gave_up))) return false;
    ++used;
    write_operand(sh.b[slot], c_step, s, lane, takes_s<KIND>(q.kind));
    fence_async_proxy();
    uint32_t t = 0;
    __syncwarp();
    if (lane == 0) t = atomicAdd(&sh.next, 1u);
    t = __shfl_sync(kFull, t, 0);
    if ((lane & 7) == 0) sh.ring[t % kRing][lane >> 3] = q;
    if (lane == 0) sh.ring_slot[t % kRing] = slot;
    __syncwarp();
    if (lane == 0) mbar_arrive(smem_addr(&sh.bar_ready[t % kRing]));
    return true;
}

// Steps of a bulk call from output `pos` on, up to output `end`.
template <int KIND, class Sh>
__device__ __forceinline__ bool produce_run(Sh& sh, const TensorArgs& a, int producer, int lane, uint64_t pos,
                                            uint64_t end) {
    uint32_t used = 0, s[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) s[q] = a.st[q];
    warp_jump(g_jwin, s, pos);
    bool ok = tables_ready(sh);
    const auto step = [&] {
        const uint64_t at = pos + (uint64_t)(lane >> 3) * kTcQuarter;
        Quarter q;
        q.out = (unsigned long long)a.out + at * elem_bytes(a.kind);
        q.count = at < end ? (uint32_t)min((uint64_t)kTcQuarter, end - at) : 0u;
        q.kind = (uint32_t)a.kind;
        return produce_step<KIND>(sh, producer, lane, used, s, q);
    };
    if (ok) {
        to_block(sh, s, lane);
        ok = step();  // the first has its operand buffer without a wait
        __syncwarp();
    }
    meet<Sh>();
    while (ok) {
        pos += kTcStep;
        if (pos >= end) return true;
        advance(s, c_step);
        ok = step();
    }
    return false;
}

// The largest i with base[i] <= ti, for four values of ti at once: the lanes of
// a group have the same ti (below base[ninst]) and search eight ways.
__device__ __forceinline__ uint32_t group_owner(const uint32_t* __restrict__ base, uint32_t ninst, uint32_t ti) {
    const int lane = threadIdx.x & 31;
    uint32_t lo = 0, hi = ninst;
    while (__any_sync(kFull, hi - lo > 1)) {
        const uint32_t step = (hi - lo + 7) / 8, c = lo + (uint32_t)(lane & 7) * step;
        const uint32_t m = (__ballot_sync(kFull, c < hi && __ldg(base + c) <= ti) >> (lane & 24)) & 255u;
        lo += (uint32_t)(31 - __clz((int)m)) * step;
        hi = min(hi, lo + step);
    }
    return lo;
}

// A producer of a batch: four streams of tiles, eight lanes each, every stream
// putting one quarter (eight blocks) of its tile into each step.  A stream's
// first tile is its index among all streams, the blocks of threads first, so
// that few tiles spread over all SMs; later ones come from the counter.
template <int KIND, class Sh>
__device__ __forceinline__ bool produce_tiles(Sh& sh, const BatchArgs& a, int producer, int lane) {
    const uint32_t streams = gridDim.x * Sh::kProducers * 4;
    uint32_t used = 0, s[8], left = 0;
    uint32_t pulled = blockIdx.x + gridDim.x * (producer * 4 + (lane >> 3));  // of the group's first lane
    Quarter q;
    q.out = 0;
    q.kind = kU32;
    bool more = true, ready = false;
#pragma unroll
    for (int i = 0; i < 8; ++i) s[i] = 1;
    for (;;) {
        while (__any_sync(kFull, more && left == 0)) {
            const uint32_t next = __shfl_sync(kFull, pulled, 0, 8);
            more = more && (left != 0 || next < a.ntiles);
            const bool take = more && left == 0;
            uint32_t n[8] = {1, 1, 1, 1, 1, 1, 1, 1};
            uint64_t k = 0;
            BatchTile t;
            BatchInst in;
            t.start = 0;
            t.inst = t.len_flags = 0;
            if (a.tiles) {
                if (take) {
                    t = a.tiles[next];
                    in = a.insts[t.inst];
                }
            } else {
                const uint32_t i = group_owner(a.tile_base, a.ninst, take ? next : 0u);
                if (take) {
                    in = a.insts[i];
                    t = derive_tile(next - a.tile_base[i], in, i, a.tile_elems);
                }
            }
            if (take) {
                const uint32_t* src = in.slot1 ? a.states + 8ull * (in.slot1 - 1) : in.st;
#pragma unroll
                for (int i = 0; i < 8; ++i) n[i] = src[i];
                k = in.offset + t.start;
                if ((lane & 7) == 0) pulled = streams + atomicAdd(a.counter, 1u);  // awaited at the next fetch
            }
            group_jump(g_jwin, n, k);
            const bool head = (t.len_flags & kTileHead) != 0;
            if (take && head && (lane & 7) == 0) {
                uint32_t st[8];
#pragma unroll
                for (int i = 0; i < 8; ++i) st[i] = n[i];
                write_head(g_jwin, in.kind, st, (char*)in.out + t.start * elem_bytes(in.kind), t.len_flags & ~kTileHead);
            }
            __syncwarp();
            if (!ready && !(ready = tables_ready(sh))) return false;
            to_block(sh, n, lane & 7);
            if (take && !head) {
#pragma unroll
                for (int i = 0; i < 8; ++i) s[i] = n[i];
                left = t.len_flags;
                q.kind = (uint32_t)in.kind;
                q.out = (unsigned long long)in.out + t.start * elem_bytes(in.kind);
            }
        }
        if (!__any_sync(kFull, left != 0)) return true;
        q.count = min(left, (uint32_t)kTcQuarter);
        if (!produce_step<KIND>(sh, producer, lane, used, s, q)) return false;
        left -= q.count;
        q.out += (unsigned long long)kTcQuarter * elem_bytes((int)q.kind);
        if (__any_sync(kFull, left != 0)) advance(s, c_quarter);
    }
}

// One block of threads: `produce(p)` runs in producer warp p and returns false
// if a wait gave up.  False if one did.  OVERLAPPED: the launch is one of
// launch_overlapped, and produce() calls meet() once.  A writer warp owns the
// tensor memory: taken in the issuing warp's branch, ahead of its loop, the bulk
// kernel ran 2^30 uint32 in 657 microseconds instead of 612, fp32 in 792 instead
// of 773.
template <int KIND, bool OVERLAPPED, class Sh, class Produce>
__device__ __forceinline__ bool run_block(Sh& sh, uint32_t* fault, Produce&& produce) {
    constexpr int kProducers = Sh::kProducers, kSlots = Sh::kSlots;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (warp == kWriters + kProducers) {
        if (lane == 0) {
            mbar_init(smem_addr(&sh.bar_tables), 1);
            for (int i = 0; i < kRing; ++i) mbar_init(smem_addr(&sh.bar_ready[i]), 1);
            for (int i = 0; i < kSlots; ++i) mbar_init(smem_addr(&sh.bar_free[i]), 1);
            for (int i = 0; i < kAccs; ++i) {
                mbar_init(smem_addr(&sh.bar_full[i]), 2);
                mbar_init(smem_addr(&sh.bar_empty[i]), kWriters / kAccs);
            }
            sh.next = sh.ended = sh.gave_up = 0;
            fence_async_proxy();
            mbar_expect_tx(smem_addr(&sh.bar_tables), sizeof(sh.a) + sizeof(sh.col));
            bulk_load(smem_addr(sh.col), g_tc_col, sizeof(sh.col), smem_addr(&sh.bar_tables));
            bulk_load(smem_addr(sh.a), g_tc_a, sizeof(sh.a), smem_addr(&sh.bar_tables));
        }
    } else if (warp >= kWriters) {
        // The operands' last K-chunk is zero throughout.
        const int p = warp - kWriters;
        for (int i = 0; i < 4; ++i)
            *reinterpret_cast<uint4*>(sh.b[2 * p + (i & 1)] + tc_half(lane + kTcCols * (i >> 1), 40, kTcN / 8)) =
                make_uint4(0u, 0u, 0u, 0u);
    } else if (warp == 0 && !OVERLAPPED) {
        tmem_alloc(smem_addr(&sh.tmem), kTmemCols);
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp < kWriters) {
        if (OVERLAPPED) {
            // Tensor memory is this block's between the end of the kernel before and
            // its own end only: a kernel before that takes tensor memory late never
            // waits for this one.  The next kernel's blocks, which may take some and
            // then wait for this kernel, start only when all blocks here own theirs.
            // With the next kernel let in at the start and tensor memory taken then,
            // calls back to back were closer up to 2^18 outputs (C ABI, microseconds:
            // 2.6 to 2.9, now 2.8 to 3.7; through Python the host takes 4), level at
            // 2^20 and further apart from there (5,000,001 fp32 8.4, now 8.2).
            after_previous_kernel();
            if (warp == 0) {
                tmem_alloc(smem_addr(&sh.tmem), kTmemCols);
                if (lane == 0) next_kernel_may_start();
                __syncwarp();
                tc_fence_before();
            }
            meet<Sh>();
            tc_fence_after();
        }
        writer<KIND>(sh, warp, lane);
    } else if (warp < kWriters + kProducers) {
        const bool ok = produce(warp - kWriters);
        __syncwarp();
        if (lane == 0 && ok && atomicAdd(&sh.ended, 1u) == kProducers - 1) {
            const uint32_t t = atomicAdd(&sh.next, 1u);
            for (int i = 0; i < 4 * kAccs; ++i) sh.ring[(t + i / 4) % kRing][i % 4].kind = kEndKind;
            mbar_arrive(smem_addr(&sh.bar_ready[t % kRing]));
        }
    } else {
        if (OVERLAPPED) {
            meet<Sh>();
            tc_fence_after();
        }
        if (lane == 0) issuer(sh);
    }
    __syncwarp();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const bool ok = !sh.gave_up;  // uniform: written before the barrier
    if (!ok) {
        if (warp == kWriters + kProducers && lane == 0) {
            // The tables' copies and the products that are under way end first, the
            // products on a barrier of their own.
            const uint32_t bar = smem_addr(&sh.ring[0][0]);
            mbar_wait_last(smem_addr(&sh.bar_tables));
            mbar_init(bar, 1);
            fence_async_proxy();
            tc_commit(bar);
            mbar_wait_last(bar);
            *reinterpret_cast<volatile uint32_t*>(fault) = 1;
            __threadfence_system();
        }
        __syncthreads();
    }
    if (warp == 0) tmem_free(sh.tmem, kTmemCols);
    return ok;
}

}  // namespace

// Producers of a bulk call (more of them, 4 to 7, measured 1 to 3 % slower).
using BulkShared = Shared<3>;

template <int KIND>
__global__ void __launch_bounds__(threads_for(BulkShared::kProducers), 1)
    k_tensor(const __grid_constant__ TensorArgs a) {
    extern __shared__ __align__(128) unsigned char raw[];
    BulkShared& sh = *reinterpret_cast<BulkShared*>(raw);
    run_block<KIND, true>(sh, a.fault, [&](int p) {
        const int lane = threadIdx.x & 31;
        // The block's quarters lo .. hi - 1, the producer's share of the steps
        // from lo on (the last of them may hold fewer than four).  Blocks of many
        // steps begin on a step (64 KB of fp64): 1,167 microseconds at 2^30 fp64,
        // 1,176 where they begin on any quarter.  Blocks of few steps share the
        // quarters out, which ends 2^24 fp64 outputs after 13.5 steps of writing, not
        // 14: 22.4, 22.8 on whole steps.  Where one passes into the other matters
        // little: from 2^25 to 2^28 outputs the two differ by under 1 %, either way
        // (fp64, whole / any: 2^26 76.7 / 77.1, 2^26 - 12,345 77.5 / 77.2, 3 * 2^25
        // 112.8 / 113.0, 2^28 295.1 / 296.3), uint32 and fp32 likewise.
        const uint64_t whole = a.quarters / gridDim.x >= 256 ? 3u : 0u;
        const uint64_t lo = a.quarters * blockIdx.x / gridDim.x & ~whole;
        const uint64_t hi = blockIdx.x + 1 == gridDim.x ? a.quarters
                                                        : a.quarters * (blockIdx.x + 1) / gridDim.x & ~whole;
        const uint64_t steps = (hi - lo + 3) / 4;
        const uint64_t first = lo + steps * p / BulkShared::kProducers * 4;
        const uint64_t last = min(hi, lo + steps * (p + 1) / BulkShared::kProducers * 4);
        bool ok = true;
        if (first >= last) meet<BulkShared>();
        else ok = produce_run<KIND>(sh, a, p, lane, a.head + first * kTcQuarter, min(a.n, a.head + last * kTcQuarter));
        if (blockIdx.x == 0 && p == 0 && lane == 0 && a.head) {
            after_previous_kernel();
            uint32_t st[8];
#pragma unroll
            for (int q = 0; q < 8; ++q) st[q] = a.st[q];
            write_head(g_jwin, a.kind, st, a.out, a.head);
        }
        return ok;
    });
}

// A batch of independent instances (BatchArgs), cut into tiles (mrg8g_tiles.h)
// that the producers take from a queue, so every instance's values equal its own
// stream.  This replaces one mrg8_cuda::mrg8_outer_32 launch per instance
// (cuda/mrg8_cuda.cu:414-436).  KIND: every instance's, or kMixed.
//
// What bounds it: one kind, the writers as in a bulk call, after the producers'
// tile setup where tiles are short; mixed kinds, the writers and their
// instruction cache.  GB300, against the recurrence kernel (microseconds): 65,536
// streams of 4,096 uint32 327 -> 179 with five producers (222 with three), 10,000
// uneven instances of three kinds (14.7 GB) 3,140 -> 2,350, 2,000 of them up to 2^20
// long 247 -> 156, 10,000 of 64 outputs 35 -> 28, 65,536 of up to 256 outputs 174 ->
// 106; smaller batches stay on that kernel (recurrence_blocks in mrg8g_tiles.h).
// Mixed batches with five producers and both quarters unrolled: 2,401 (2,443 as kept,
// before fp32 was rounded with eight low bits), but 165 and up to 229 in the smaller
// ones; with the code of five kinds instead of three, and no order of kinds, 2,760.
template <int KIND>
using BatchShared = Shared<KIND == kMixed ? 3 : 5>;

template <int KIND>
__global__ void __launch_bounds__(threads_for(BatchShared<KIND>::kProducers), 1)
    k_tensor_batch(const __grid_constant__ BatchArgs a) {
    extern __shared__ __align__(128) unsigned char raw[];
    BatchShared<KIND>& sh = *reinterpret_cast<BatchShared<KIND>*>(raw);
    if (a.times && blockIdx.x == 0 && threadIdx.x == 0) a.times[0] = global_ns();
    run_block<KIND, false>(sh, a.fault, [&](int p) { return produce_tiles<KIND>(sh, a, p, threadIdx.x & 31); });
    leave_queue(a);
}

#define MRG8G_EACH_KIND(F) F(kU32) F(kF64Orig) F(kF64Shift) F(kF32Orig) F(kF32Shift)

cudaError_t prepare_tensor() {
    constexpr auto kAttr = cudaFuncAttributeMaxDynamicSharedMemorySize;
    cudaError_t e = cudaFuncSetAttribute(k_tensor_batch<kMixed>, kAttr, (int)sizeof(BatchShared<kMixed>));
#define MRG8G_PREPARE(K)                                                                                \
    if (e == cudaSuccess) e = cudaFuncSetAttribute(k_tensor<K>, kAttr, (int)sizeof(BulkShared));         \
    if (e == cudaSuccess) e = cudaFuncSetAttribute(k_tensor_batch<K>, kAttr, (int)sizeof(BatchShared<K>));
    MRG8G_EACH_KIND(MRG8G_PREPARE)
#undef MRG8G_PREPARE
    return e;
}

cudaError_t launch_tensor(const TensorArgs& a, int sms, cudaStream_t st) {
    constexpr int threads = threads_for(BulkShared::kProducers);
    const uint64_t steps = (a.quarters + 3) / 4;
    const int blocks = (int)(steps < (uint64_t)sms ? (steps ? steps : 1) : (uint64_t)sms);
    switch (a.kind) {
#define MRG8G_LAUNCH(K) \
    case K: return launch_overlapped(k_tensor<K>, blocks, threads, sizeof(BulkShared), st, a);
        MRG8G_EACH_KIND(MRG8G_LAUNCH)
#undef MRG8G_LAUNCH
    }
    return cudaErrorInvalidValue;
}

template <int KIND>
static void launch_batch_t(const BatchArgs& a, int blocks, cudaStream_t st) {
    k_tensor_batch<KIND><<<blocks, threads_for(BatchShared<KIND>::kProducers), sizeof(BatchShared<KIND>), st>>>(a);
}

cudaError_t launch_tensor_batch(const BatchArgs& a, int kind, int sms, cudaStream_t st) {
    const int blocks = (int)(a.ntiles < (uint32_t)sms ? a.ntiles : (uint32_t)sms);
    switch (kind) {
#define MRG8G_LAUNCH(K) \
    case K: launch_batch_t<K>(a, blocks, st); break;
        MRG8G_EACH_KIND(MRG8G_LAUNCH)
#undef MRG8G_LAUNCH
    default: launch_batch_t<kMixed>(a, blocks, st);
    }
    return cudaGetLastError();
}

}  // namespace mrg8g
