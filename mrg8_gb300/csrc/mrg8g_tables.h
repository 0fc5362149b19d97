// mrg8g_tables.h -- host-generated constants of the MRG8 recurrence.
//
// The generator state is s = (S[n-1], ..., S[n-8]) (newest first, as in
// original/mrg8.h:49) and one step is s' = A s with A the companion matrix:
// row 0 holds the coefficients a_1..a_8 (original/mrg8.cpp:16-18) and the
// sub-diagonal holds ones.  Everything here is computed on the host at load
// time; nothing is read from files.
#pragma once
#include <stdint.h>

#if defined(__CUDACC__)
#define MRG8G_HDC __host__ __device__
#else
#define MRG8G_HDC
#endif

namespace mrg8g {

constexpr int kNumJump = 247;   // A^(2^i), i = 0..246 (jump_matrix.txt depth)

// Byte-window jump table of the device: jwin[w * 255 + j - 1] = A^(j 256^w)
// for byte position w = 0..7 and byte value j = 1..255, so a 64-bit jump is
// at most eight matrix-vector products (one per non-zero byte of the offset)
// instead of one per set bit.  jwin[0] = A (row 0 = the coefficients).
constexpr int kJumpBytes = 8;
constexpr int kJumpWinMats = kJumpBytes * 255;

// Lane layouts of the bulk kernels: a warp of 32 lanes, each lane writing V
// consecutive outputs per row, so consecutive rows of one lane are d = 32 V
// positions apart.  Supported V: 1, 2, 4 -> d = 32, 64, 128.
constexpr int kNumLayouts = 3;
MRG8G_HDC constexpr int layout_index(int V) { return V == 1 ? 0 : (V == 2 ? 1 : 2); }
MRG8G_HDC constexpr int layout_stride(int li) { return 32 << li; }
// Offsets (in u32 words) of each layout's window table inside one array.
MRG8G_HDC constexpr int win_offset(int li) { return li == 0 ? 0 : (li == 1 ? 32 * 64 : 96 * 64); }
constexpr int kWinWords = (32 + 64 + 128) * 64;

// Decimated recurrence.  The stride-d subsequence T_j = S[o + d j] of any
// MRG8 stream satisfies T_j = sum_k beta_k T_{j-k} (k = 1..8), where
// x^8 - sum beta_k x^(8-k) is the characteristic polynomial of A^d
// (Cayley-Hamilton).  For the kernels the coefficients are stored signed,
// c_k = beta_k or beta_k - p (|c_k| < 2^30), and the kernels keep the lagged
// values as x = S - 1 in [0, p-1] (`leap`); then
//     a = K1 + sum_k c_k x_{j-k}
// lies in [0, 2^64 - 1) and a == S_j - 1 (mod p), where K1 == sum_k c_k - 1
// (mod p) is the smallest such constant keeping a >= 0.  With the lagged
// values kept as s = S mod p instead (`leap_mod`, the fp64 ORIGINAL outputs), the
// same coefficients and K1 == 0 (mod p) give a == S_j (mod p).
struct LeapCoef {
    int32_t c[8];
    uint64_t K1;
};

// Block form of the tensor-core kernel (mrg8g_tensor.cu).  A block is 256
// outputs of a stream at constant distances from its start B; all of them follow
// from the state s there by constant rows, S[B + m - 1] = e_0^T A^m s, so with the
// 8 state words cut into 32 bytes and every coefficient into three signed
// 11-bit limbs a block is an exact fp16 product with fp32 sums.
//   B operand, rows l and kTcCols + l of kTcK halves for block l, from its
//     state and from the state one output later: [0, 32) byte i of word q at
//     4 q + i, less 128; [32] 4096; [33] 1; [34] 1 for S, 0 for S - 1; rest 0.
//   A operand, matrix j of kTcM rows of kTcK halves (limb j; row r gives
//     outputs tc_row(r) and the next with a block's two rows, m = tc_row(r) + 1): [0, 32)
//     limb j of 2 u_m[q] 2^(8 i) mod p; [32] 3072; [33] limb j of the row's
//     constant; [34] 1 for j = 0.  The representatives mod p are the even ones
//     below p in magnitude, v = 2 l_0 + 2^11 l_1 + 2^22 l_2.
// Column 32 adds 1.5 * 2^23 to every sum, so that the fp32 word of a sum P is
// 0x4B400000 + P, and with the row constants
//   W = 2 w_0 + 2^11 w_1 + 2^22 w_2 == 2 (S - 1) (mod p), or 2 S,
// for the three words of an output.  W is even and 2^31 == 1, so with
// V = 2^11 w_1 + 2^22 w_2 its half is (V >> 32) + (V mod 2^32) / 2 + w_0 (mod p),
// below 2 p.  Every |P| < 2^22 (checked when the table is built), so all sums
// are integers below 2^24: exact in fp32.
constexpr int kTcBlock = 256;             // outputs per block
constexpr int kTcQuarter = 8 * kTcBlock;  // outputs of eight blocks
constexpr int kTcM = 128, kTcK = 48;      // rows and depth of an A matrix
constexpr int kTcMats = 3;
constexpr int kTcCols = 32;               // blocks per step, one lane each
constexpr int kTcN = 2 * kTcCols;         // rows of the B operand
constexpr int kTcStep = kTcBlock * kTcCols;  // outputs per step
constexpr int kTcMatHalves = kTcM * kTcK;
// Where outputs lie.  Block l starts tc_block(l) outputs into its step, and row
// r of the A operand gives its outputs tc_row(r) and the next: the eight blocks
// of a quarter interleave, so that the 32 rows of one warp and the eight blocks
// are 512 consecutive outputs.
MRG8G_HDC constexpr int tc_block(int l) { return kTcQuarter * (l >> 3) + 64 * (l & 7); }
MRG8G_HDC constexpr int tc_row(int r) { return 512 * (r >> 5) + 2 * (r & 31); }
// Half (r, k) of a matrix or operand with `groups` groups of eight rows: the
// 16-byte K-chunks of eight rows are 128 contiguous bytes, groups next, chunks
// last (K-major without swizzle).
MRG8G_HDC constexpr int tc_half(int r, int k, int groups) {
    return ((k >> 3) * groups + (r >> 3)) * 64 + (r & 7) * 8 + (k & 7);
}

// State advance with a constant matrix: row r of the new state is
// K[r] + sum_q c[8 r + q] s_q reduced mod p (c centred, K[r] == 0 mod p keeps
// the sum in [0, 2^64) for words s_q in [0, p]).
struct StepCoef {
    int32_t c[64];
    uint64_t K[8];
    int32_t c1[8];  // row 0 of A: the next output
    uint64_t K1;
};

struct TensorTables {
    uint16_t a[kTcMats * kTcMatHalves];  // fp16, each matrix laid out by tc_half
    // A^(tc_block(l)) for lane l = 0..31: word (r, c) at [(r * 8 + c) / 4][l][c % 4].
    uint32_t col[16 * 32 * 4];
    StepCoef step;                       // A^(kTcStep)
    StepCoef quarter;                    // A^(kTcQuarter)
};

struct HostTables {
    // jump[i][r*8+c] = A^(2^i)(r, c), row-major, canonical residues.
    uint32_t jump[kNumJump][64];
    // Byte windows (above), row-major like jump: 2040 matrices, 522,240 bytes.
    uint32_t jwin[kJumpWinMats][64];
    // Window tables, per layout li with stride d: win[off + (o*8 + j)*8 + c]
    // is column c of the row vector e_0^T A^(o + 1 + d j), o in [0, d),
    // j in [0, 8): S[B + o + d j] = win_row . s_B for a state s_B taken at
    // stream position B.
    uint32_t win[kWinWords];
    // Row-block steps of the layouts: dstep[li][j - 1] = A^(d j) for
    // d = layout_stride(li), j = 1..7 (the states at the starts of a warp's
    // first eight rows, from which its lanes form their windows).
    uint32_t dstep[kNumLayouts][7][64];
    LeapCoef leap[kNumLayouts];
    LeapCoef leap_mod[kNumLayouts];
    TensorTables tc;
};

// Built once (thread-safe) on first use.
const HostTables& host_tables();

// Row-major 8x8 product mod p, canonical entries.
void matmul_mod(const uint32_t* X, const uint32_t* Y, uint32_t* C);

// new_state = A^k state by per-bit matrix-vector products with the table
// (knl/mrg8.h:212-238).  Entries come back in [1, p] (0 only for an all-zero
// contribution), as bigDotProd does.
void jump_matvec(const uint32_t st[8], uint64_t k, uint32_t out[8]);

// Same over a 200-bit little-endian bit array (bits[i] != 0 -> set).
void jump_matvec_bits(const uint32_t st[8], const short bits[200], uint32_t out[8]);

// original/mrg8.cpp:104-176 exactly: J = product of A^(2^i) over the set bits
// formed with bigDotProd, then state <- J state.
void jump_exact_bits(const uint32_t st[8], const short bits[200], uint32_t out[8]);

// Sequential recurrence on the host for a handful of steps (state update of
// original/mrg8.cpp:197-222); outputs optional.
void step_host(uint32_t st[8], uint64_t n, uint32_t* out);

// seeding of original/mrg8.cpp:180-194.
void mcg64ni(uint32_t seed, uint32_t st[8]);

}  // namespace mrg8g
