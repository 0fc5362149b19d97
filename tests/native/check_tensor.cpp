// check_tensor.cpp -- CPU check of the tensor-core kernel's tables
// (TensorTables in mrg8g_tables.h) with the kernel's own arithmetic.
//
//   check_tensor conv
//       f64_bits_fma(v) == the word of double(v) * (1.0 / (2^31 - 1)) for every
//       v in [0, 2^31 - 1] but those of f64_fma_rare, at most 1024; the same of
//       f32_bits_fma and (float) of it, but for those of f32_fma_rare, at most 4096.
//   check_tensor <stream.bin> <s0..s7>
//       stream.bin holds the oracle's outputs S[0..N), N = two steps, from
//       state s.  For both steps and every lane: the lane's start state (`col`,
//       then `step`), its bytes as the fp16 operand, its products summed as
//       integers, each sum inside the range that makes its fp32 word exact, and
//       the output put together from the three words as S - 1 and as S.
#include <atomic>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <thread>
#include <vector>

#include "mrg8g_arith.cuh"
#include "mrg8g_tables.h"

using namespace mrg8g;

static int half_value(uint16_t h) {
    if ((h & 0x7FFF) == 0) return 0;
    const int e = ((h >> 10) & 31) - 25, f = 1024 + (h & 1023);
    const int v = e >= 0 ? f << e : f >> -e;
    return h & 0x8000 ? -v : v;
}

int main(int argc, char** argv) {
    if (argc == 2 && !std::strcmp(argv[1], "conv")) {
        std::atomic<long> bad{0}, rare{0}, rare32{0};
        std::vector<std::thread> team;
        for (uint32_t part = 0; part < 8; ++part)  // v = part (mod 8): the host is slow on the tiny floats
            team.emplace_back([&, part] {
                const double rnorm = 1.0 / (double)kP;
                for (uint64_t v = part; v <= kP; v += 8) {
                    const double u = (double)v * rnorm;
                    uint64_t w;
                    uint32_t xn;
                    std::memcpy(&w, &u, 8);
                    const uint64_t got = f64_bits_fma((uint32_t)v, xn);
                    if (f64_fma_rare(xn)) ++rare;
                    else if (got != w) ++bad;
                    const float f = (float)u;
                    float fh;
                    uint32_t w32;
                    std::memcpy(&w32, &f, 4);
                    const uint32_t got32 = f32_bits_fma((uint32_t)v, fh);
                    if (f32_fma_rare(std::fabs(fh - 0.5f))) ++rare32;
                    else if (got32 != w32) ++bad;
                }
            });
        for (std::thread& t : team) t.join();
        std::printf("bad=%ld rare=%ld %ld\n", bad.load(), rare.load(), rare32.load());
        return bad != 0 || rare > 1024 || rare32 > 4096;
    }
    if (argc != 10) return 2;
    FILE* f = std::fopen(argv[1], "rb");
    if (!f) return 2;
    std::vector<uint32_t> S(2 * kTcStep);
    if (std::fread(S.data(), 4, S.size(), f) != S.size()) return 2;
    std::fclose(f);
    uint32_t s[8];
    for (int q = 0; q < 8; ++q) s[q] = (uint32_t)std::strtoul(argv[2 + q], nullptr, 10);
    const TensorTables& tc = host_tables().tc;
    uint32_t st[kTcCols][8];
    for (int l = 0; l < kTcCols; ++l)
        for (int r = 0; r < 8; ++r) {
            uint32_t m[8];
            for (int c = 0; c < 8; ++c) m[c] = tc.col[(((r * 8 + c) >> 2) * 32 + l) * 4 + (c & 3)];
            st[l][r] = dot8_ref(m, s);
        }
    long bad = 0, wide = 0;
    uint32_t row[8];
    for (int step = 0; step < 2; ++step)
        for (int l = 0; l < kTcCols; ++l) {
            for (int tt = 0; tt < 2; ++tt) {
                if (tt) {  // the state one output later
                    uint64_t acc = tc.step.K1;
                    for (int q = 0; q < 8; ++q) acc = mad_wide_s32(tc.step.c1[q], st[l][q], acc);
                    std::memcpy(row + 1, st[l], 28);
                    row[0] = reduce_acc(acc);
                } else {
                    std::memcpy(row, st[l], 32);
                }
                for (int r = 0; r < kTcM; ++r) {
                    uint32_t word[2][3];
                    for (int mod = 0; mod < 2; ++mod)  // 0: S - 1, 1: S
                        for (int j = 0; j < 3; ++j) {
                            const uint16_t* a = tc.a + j * kTcMatHalves;
                            long sum = 0;
                            for (int k = 0; k < kTcK; ++k) {
                                const int b = k < 32 ? (int)((row[k >> 2] >> (8 * (k & 3))) & 255) - 128
                                              : k == 32 ? 4096 : k == 33 ? 1 : k == 34 ? mod : 0;
                                sum += (long)half_value(a[tc_half(r, k, kTcM / 8)]) * b;
                            }
                            wide += sum < 1 << 23 || sum >= 1 << 24;
                            word[mod][j] = 0x4B400000u + (uint32_t)(sum - (3 << 22));  // of the fp32 sum
                        }
                    const uint32_t want = S[step * kTcStep + tc_block(l) + tc_row(r) + tt];
                    for (int mod = 0; mod < 2; ++mod) {
                        const uint64_t v = (uint64_t)word[mod][1] * (1u << 11) + (uint64_t)word[mod][2] * (1u << 22);
                        const uint32_t y = (uint32_t)(v >> 32) + ((uint32_t)v >> 1) + word[mod][0], z = y - kP;
                        bad += (uint64_t)(uint32_t)(v >> 32) + ((uint32_t)v >> 1) + word[mod][0] >= 2ull * kP;
                        if (mod) bad += (uint32_t)((int32_t)y > (int32_t)z ? y : z) != want;
                        else bad += (y < z ? y : z) != want - 1;
                    }
                }
            }
            uint32_t n[8];
            for (int r = 0; r < 8; ++r) {
                uint64_t acc = tc.step.K[r];
                for (int q = 0; q < 8; ++q) acc = mad_wide_s32(tc.step.c[r * 8 + q], st[l][q], acc);
                n[r] = reduce_acc(acc);
            }
            for (int r = 0; r < 8; ++r) st[l][r] = n[r];
        }
    std::printf("bad=%ld wide=%ld\n", bad, wide);
    return bad || wide;
}
