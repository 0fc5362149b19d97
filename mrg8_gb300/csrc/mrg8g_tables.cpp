// mrg8g_tables.cpp -- host generation of the jump tables, window tables and
// decimated-recurrence coefficients (see mrg8g_tables.h).
#include "mrg8g_tables.h"

#include <cstring>
#include <mutex>
#include <stdexcept>

#include "mrg8g_arith.cuh"

namespace mrg8g {

// original/mrg8.cpp:16-18.
static const uint32_t kCoef[8] = {1089656042u, 1906537547u, 1764115693u, 1304127872u,
                                  189748160u,  1984088114u, 626062218u,  1927846343u};

static uint32_t mulmod(uint32_t a, uint32_t b) { return (uint32_t)(((uint64_t)a * b) % kP); }
static uint32_t addmod(uint32_t a, uint32_t b) {
    uint32_t s = a + b;  // both < 2^31
    return s >= kP ? s - kP : s;
}
static uint32_t submod(uint32_t a, uint32_t b) { return a >= b ? a - b : a + kP - b; }
static uint32_t powmod(uint32_t a, uint64_t e) {
    uint64_t r = 1, x = a % kP;
    while (e) {
        if (e & 1) r = r * x % kP;
        x = x * x % kP;
        e >>= 1;
    }
    return (uint32_t)r;
}
static uint32_t invmod(uint32_t a) { return powmod(a, kP - 2); }  // p prime

void matmul_mod(const uint32_t* X, const uint32_t* Y, uint32_t* C) {
    uint32_t T[64];
    for (int r = 0; r < 8; ++r)
        for (int c = 0; c < 8; ++c) {
            uint64_t acc = 0;
            for (int q = 0; q < 8; ++q) acc += ((uint64_t)X[r * 8 + q] * Y[q * 8 + c]) % kP;
            T[r * 8 + c] = (uint32_t)(acc % kP);
        }
    std::memcpy(C, T, sizeof(T));
}

static void matvec_mod(const uint32_t* M, const uint32_t* v, uint32_t* out) {
    uint32_t t[8];
    for (int r = 0; r < 8; ++r) {
        uint64_t acc = 0;
        for (int q = 0; q < 8; ++q) acc += ((uint64_t)M[r * 8 + q] * v[q]) % kP;
        t[r] = (uint32_t)(acc % kP);
    }
    std::memcpy(out, t, sizeof(t));
}

// Solve C beta = rhs (mod p) for an invertible 8x8 C (Gauss-Jordan).
static bool solve8(uint32_t C[8][9], uint32_t beta[8]) {
    for (int col = 0; col < 8; ++col) {
        int piv = -1;
        for (int r = col; r < 8; ++r)
            if (C[r][col]) { piv = r; break; }
        if (piv < 0) return false;
        if (piv != col)
            for (int c = 0; c < 9; ++c) std::swap(C[piv][c], C[col][c]);
        const uint32_t inv = invmod(C[col][col]);
        for (int c = 0; c < 9; ++c) C[col][c] = mulmod(C[col][c], inv);
        for (int r = 0; r < 8; ++r) {
            if (r == col || !C[r][col]) continue;
            const uint32_t f = C[r][col];
            for (int c = 0; c < 9; ++c) C[r][c] = submod(C[r][c], mulmod(f, C[col][c]));
        }
    }
    for (int r = 0; r < 8; ++r) beta[r] = C[r][8];
    return true;
}

// beta_k with M^8 v = sum_k beta_k M^(8-k) v for every v (characteristic
// polynomial of M, which is irreducible for powers of A, so any non-zero v is
// cyclic).  Solved on v = e_0 and checked on a second vector.
static void charpoly_coeffs(const uint32_t* M, uint32_t beta[8]) {
    uint32_t pw[9][8];
    std::memset(pw, 0, sizeof(pw));
    pw[0][0] = 1;
    for (int i = 1; i <= 8; ++i) matvec_mod(M, pw[i - 1], pw[i]);
    uint32_t C[8][9];
    for (int r = 0; r < 8; ++r) {
        for (int k = 1; k <= 8; ++k) C[r][k - 1] = pw[8 - k][r];
        C[r][8] = pw[8][r];
    }
    if (!solve8(C, beta)) throw std::runtime_error("mrg8g: singular Krylov matrix");
    uint32_t q[9][8];
    for (int r = 0; r < 8; ++r) q[0][r] = (uint32_t)(r * 7919 + 13);
    for (int i = 1; i <= 8; ++i) matvec_mod(M, q[i - 1], q[i]);
    for (int r = 0; r < 8; ++r) {
        uint32_t acc = 0;
        for (int k = 1; k <= 8; ++k) acc = addmod(acc, mulmod(beta[k - 1], q[8 - k][r]));
        if (acc != q[8][r]) throw std::runtime_error("mrg8g: characteristic polynomial check failed");
    }
}

// K1 == sum_k c_k - 1 (mod p) for lags x = S - 1, K1 == 0 (mod p) for lags
// s = S mod p (mod_lags).
static LeapCoef make_leap(const uint32_t beta[8], bool mod_lags) {
    LeapCoef lc;
    int64_t csum = 0;
    unsigned __int128 negsum = 0, possum = 0;
    for (int k = 0; k < 8; ++k) {
        const int64_t c = beta[k] <= (kP - 1) / 2 ? (int64_t)beta[k] : (int64_t)beta[k] - (int64_t)kP;
        lc.c[k] = (int32_t)c;
        csum += c;
        if (c < 0) negsum += (unsigned __int128)(-c);
        else possum += (unsigned __int128)c;
    }
    // K1 == cmod (mod p), the smallest such value >= negsum (p - 1), so that
    // K1 + sum c_k x_k (x_k in [0, p-1]) stays in [0, 2^64 - 1).
    const uint64_t cmod = mod_lags ? 0 : (uint64_t)(((csum - 1) % (int64_t)kP + (int64_t)kP) % (int64_t)kP);
    const unsigned __int128 base = negsum * (kP - 1);
    const uint64_t bmod = (uint64_t)(base % kP);
    const unsigned __int128 K1 = base + (cmod + kP - bmod) % kP;
    const unsigned __int128 top = K1 + possum * (kP - 1);
    if (top >= ~(unsigned __int128)0 >> 64) throw std::runtime_error("mrg8g: accumulator range exceeds 64 bits");
    lc.K1 = (uint64_t)K1;
    return lc;
}

static int64_t centred(uint32_t v) { return v <= (kP - 1) / 2 ? (int64_t)v : (int64_t)v - (int64_t)kP; }

// fp16 word of an integer that fp16 holds exactly.
static uint16_t half_of(int v) {
    if (v == 0) return 0;
    const uint16_t sign = v < 0 ? 0x8000u : 0u;
    const uint32_t a = (uint32_t)(v < 0 ? -v : v);
    const int e = 31 - __builtin_clz(a);
    const uint32_t frac = e <= 10 ? a << (10 - e) : a >> (e - 10);
    if (e > 10 && (frac << (e - 10)) != a) throw std::runtime_error("mrg8g: integer not exact in fp16");
    return (uint16_t)(sign | ((uint32_t)(e + 15) << 10) | (frac & 0x3FFu));
}

// The even representative of v in (-p, p).
static int64_t even_residue(uint32_t v) { return v & 1 ? (int64_t)v - (int64_t)kP : (int64_t)v; }

// v = 2 l[0] + 2^11 l[1] + 2^22 l[2] for even v, l[0] in [-512, 511], l[1] in
// [-1024, 1023].
static void limbs11(int64_t v, int l[3]) {
    for (int j = 0; j < 2; ++j) {
        l[j] = (int)((v + 1024) & 2047) - 1024;
        v = (v - l[j]) >> 11;
    }
    l[0] /= 2;
    l[2] = (int)v;
}

// Centred coefficients of a row and the smallest multiple of p that keeps the
// sum in [0, 2^64) for any words in [0, p].
static uint64_t centred_row(const uint32_t* row, int32_t* c) {
    unsigned __int128 neg = 0, pos = 0;
    for (int q = 0; q < 8; ++q) {
        const int64_t v = centred(row[q]);
        c[q] = (int32_t)v;
        if (v < 0) neg += (unsigned __int128)(-v);
        else pos += (unsigned __int128)v;
    }
    if ((neg + pos) * kP >= ~(unsigned __int128)0 >> 64) throw std::runtime_error("mrg8g: step sum exceeds 64 bits");
    return (uint64_t)(neg * kP);
}

static StepCoef make_step(const uint32_t* M) {
    StepCoef s;
    for (int r = 0; r < 8; ++r) s.K[r] = centred_row(M + r * 8, s.c + r * 8);
    s.K1 = centred_row(kCoef, s.c1);
    return s;
}

// The tensor-core kernel's tables from the rows u[m] = e_0^T A^m (m = 1..256).
static void build_tensor(HostTables& t, uint32_t (*u)[8]) {
    TensorTables& tc = t.tc;
    std::memset(tc.a, 0, sizeof(tc.a));
    // The fp32 word of 1.5 * 2^23, in each of the three weighted words.
    const uint32_t E = (uint32_t)((0x4B400000ull * (2 + (1ull << 11)) + (0x4B400000ull % kP) * ((1ull << 22) % kP)) % kP);
    for (int r = 0; r < kTcM; ++r) {
        const uint32_t* row = u[tc_row(r) + 1];
        int64_t mag[3] = {0, 0, 0};
        uint32_t csum = 0;
        int l[3];
        for (int k = 0; k < 32; ++k) {
            const uint32_t c = mulmod(row[k >> 2], (uint32_t)((2ull << (8 * (k & 3))) % kP));
            csum = addmod(csum, c);
            limbs11(even_residue(c), l);
            for (int j = 0; j < kTcMats; ++j) {
                mag[j] += 128 * (l[j] < 0 ? -l[j] : l[j]);
                tc.a[j * kTcMatHalves + tc_half(r, k, kTcM / 8)] = half_of(l[j]);
            }
        }
        limbs11(even_residue(submod(submod(mulmod(128, csum), E), 2)), l);
        for (int j = 0; j < kTcMats; ++j) {
            if (mag[j] + (l[j] < 0 ? -l[j] : l[j]) + 1 >= 1 << 22)
                throw std::runtime_error("mrg8g: limb sum exceeds 22 bits");
            uint16_t* a = tc.a + j * kTcMatHalves;
            a[tc_half(r, 32, kTcM / 8)] = half_of(3072);
            a[tc_half(r, 33, kTcM / 8)] = half_of(l[j]);
            a[tc_half(r, 34, kTcM / 8)] = half_of(j == 0);
        }
    }
    // Per-lane block starts: jump[6] = A^64, jump[11] = A^2048.
    uint32_t G[64], M[64];
    std::memset(G, 0, sizeof(G));
    for (int r = 0; r < 8; ++r) G[r * 8 + r] = 1;
    for (int l = 0; l < kTcCols; ++l) {
        if (l % 8 == 0) std::memcpy(M, G, sizeof(M));
        for (int i = 0; i < 64; ++i) tc.col[((i >> 2) * 32 + l) * 4 + (i & 3)] = M[i];
        matmul_mod(M, t.jump[6], M);
        if (l % 8 == 7) matmul_mod(G, t.jump[11], G);
    }
    tc.step = make_step(G);  // A^(4 * 2048)
    tc.quarter = make_step(t.jump[11]);
}

static void build(HostTables& t) {
    uint32_t M[64];
    std::memset(M, 0, sizeof(M));
    for (int c = 0; c < 8; ++c) M[c] = kCoef[c];
    for (int r = 1; r < 8; ++r) M[r * 8 + r - 1] = 1;
    for (int i = 0; i < kNumJump; ++i) {
        std::memcpy(t.jump[i], M, sizeof(M));
        matmul_mod(M, M, M);
    }
    for (int w = 0; w < kJumpBytes; ++w) {
        std::memcpy(t.jwin[w * 255], t.jump[8 * w], sizeof(M));  // A^(256^w)
        for (int j = 2; j <= 255; ++j) matmul_mod(t.jwin[w * 255 + j - 2], t.jump[8 * w], t.jwin[w * 255 + j - 1]);
    }
    // Row vectors u_m = e_0^T A^m, m = 1..2048.
    static uint32_t u[kTcQuarter + 1][8];
    for (int c = 0; c < 8; ++c) u[1][c] = kCoef[c];
    for (int m = 2; m <= kTcQuarter; ++m)
        for (int c = 0; c < 8; ++c)  // (u A)[c] = u[0] a_c + u[c+1]
            u[m][c] = addmod(mulmod(u[m - 1][0], kCoef[c]), c < 7 ? u[m - 1][c + 1] : 0u);
    for (int li = 0; li < kNumLayouts; ++li) {
        const int d = layout_stride(li);
        uint32_t* w = t.win + win_offset(li);
        for (int o = 0; o < d; ++o)
            for (int j = 0; j < 8; ++j)
                for (int c = 0; c < 8; ++c) w[(o * 8 + j) * 8 + c] = u[o + 1 + d * j][c];
        std::memcpy(t.dstep[li][0], t.jump[5 + li], sizeof(M));  // A^d = A^(2^(5+li))
        for (int j = 2; j <= 7; ++j) matmul_mod(t.dstep[li][j - 2], t.jump[5 + li], t.dstep[li][j - 1]);
        uint32_t beta[8];
        charpoly_coeffs(t.jump[5 + li], beta);
        t.leap[li] = make_leap(beta, false);
        t.leap_mod[li] = make_leap(beta, true);
    }
    build_tensor(t, u);
}

const HostTables& host_tables() {
    static HostTables t;  // static storage: built once, no heap
    static std::once_flag once;
    std::call_once(once, [] { build(t); });
    return t;
}

void mcg64ni(uint32_t seed, uint32_t st[8]) {
    uint64_t x = seed == 0 ? 97531u : seed;
    for (int k = 0; k < 8; ++k) {
        x = 6364136223846793005ull * x;
        st[k] = (uint32_t)((x >> 32) >> 1);
    }
}

static void matvec_ref(const uint32_t* Mrow, const uint32_t* v, uint32_t* out) {
    uint32_t t[8];
    for (int r = 0; r < 8; ++r) t[r] = dot8_ref(Mrow + r * 8, v);
    std::memcpy(out, t, sizeof(t));
}

void jump_matvec(const uint32_t st[8], uint64_t k, uint32_t out[8]) {
    const HostTables& t = host_tables();
    uint32_t cur[8];
    std::memcpy(cur, st, sizeof(cur));
    for (int i = 0; i < 64; ++i)
        if ((k >> i) & 1u) matvec_ref(t.jump[i], cur, cur);
    std::memcpy(out, cur, sizeof(cur));
}

void jump_matvec_bits(const uint32_t st[8], const short bits[200], uint32_t out[8]) {
    const HostTables& t = host_tables();
    uint32_t cur[8];
    std::memcpy(cur, st, sizeof(cur));
    for (int i = 0; i < 200; ++i)
        if (bits[i]) matvec_ref(t.jump[i], cur, cur);
    std::memcpy(out, cur, sizeof(cur));
}

void jump_exact_bits(const uint32_t st[8], const short bits[200], uint32_t out[8]) {
    const HostTables& t = host_tables();
    uint32_t J[64], T[64], col[8];
    for (int r = 0; r < 8; ++r)
        for (int c = 0; c < 8; ++c) J[r * 8 + c] = (r == c);
    for (int nb = 0; nb < 200; ++nb) {
        if (!bits[nb]) continue;
        for (int c = 0; c < 8; ++c) {
            for (int q = 0; q < 8; ++q) col[q] = t.jump[nb][q * 8 + c];
            for (int r = 0; r < 8; ++r) T[r * 8 + c] = dot8_ref(J + r * 8, col);
        }
        std::memcpy(J, T, sizeof(T));
    }
    matvec_ref(J, st, out);
}

void step_host(uint32_t st[8], uint64_t n, uint32_t* out) {
    for (uint64_t i = 0; i < n; ++i) {
        const uint32_t z = dot8_ref(kCoef, st);
        std::memmove(st + 1, st, 7 * sizeof(uint32_t));
        st[0] = z;
        if (out) out[i] = z;
    }
}

}  // namespace mrg8g
