// check_waits.cpp -- what a wait that gave up inside a kernel leads to, with the
// library's own objects linked in.
//
//   check_waits host
//       The device's error word is set, as such a kernel does: every call that
//       launches or waits returns MRG8G_ERR_TIMEOUT and leaves handles as they
//       were, and all work again once the word is cleared.
#include <cuda_runtime.h>

#include <cstdio>
#include <cstring>
#include <vector>

#include "mrg8g.h"
#include "mrg8g_internal.h"
#include "mrg8g_runtime.h"

static int bad = 0;

#define EXPECT(call, want)                                                                            \
    do {                                                                                              \
        const long long got_ = (long long)(call), want_ = (long long)(want);                          \
        if (got_ != want_) std::printf("line %d: %s is %lld, not %lld\n", __LINE__, #call, got_, want_), ++bad; \
    } while (0)

static void set_word(uint32_t v) { EXPECT(cudaMemcpy(mrg8g::device_fault(), &v, sizeof(v), cudaMemcpyDefault), 0); }

static int check_host() {
    mrg8g_generator* g = nullptr;
    EXPECT(mrg8g_create(5, &g), 0);
    double* d = nullptr;
    uint64_t* offs = nullptr;
    uint32_t *states = nullptr, st[8], after[8];
    EXPECT(cudaMalloc(&d, 8 << 20), 0);
    EXPECT(cudaMalloc(&offs, 64), 0);
    EXPECT(cudaMemset(offs, 1, 64), 0);
    EXPECT(cudaMalloc(&states, 8 * 32), 0);
    EXPECT(mrg8g_get_state(g, st), 0);
    std::vector<double> host(100000);
    mrg8g_instance in{};
    std::memcpy(in.state, st, sizeof(st));
    in.n = 5000;
    in.out = d;
    in.kind = MRG8G_F64_SHIFTED;
    mrg8g_batch* b = nullptr;
    EXPECT(mrg8g_batch_create(&in, 1, nullptr, &b), 0);
    mrg8g_server_config cfg{};
    cfg.budget_bytes = 16 << 20;
    mrg8g_server* sv = nullptr;
    EXPECT(mrg8g_server_create(&cfg, &sv), 0);
    const auto calls = [&](int want) {
        EXPECT(mrg8g_generate(g, d, 10, MRG8G_U32, nullptr), want);
        EXPECT(mrg8g_generate(g, d, 5000, MRG8G_F64_ORIGINAL, nullptr), want);
        EXPECT(mrg8g_generate_host(g, host.data(), 10, MRG8G_U32), want);
        EXPECT(mrg8g_generate_host(g, host.data(), host.size(), MRG8G_F64_ORIGINAL), want);
        EXPECT(mrg8g_generate_from_state(st, 3, d, 10, MRG8G_U32, nullptr), want);
        EXPECT(mrg8g_generate_each(&in, 1, nullptr), want);
        EXPECT(mrg8g_jump_states(st, offs, states, 8, nullptr), want);
        EXPECT(mrg8g_convert((const uint32_t*)d, d + 10000, 100, MRG8G_F64_SHIFTED, nullptr), want);
        EXPECT(mrg8g_batch_launch(b, nullptr), want);
        EXPECT(mrg8g_batch_generate_noalloc(&in, 1, nullptr), want);
        EXPECT(mrg8g_stream_sync(nullptr), want);
    };
    calls(0);
    EXPECT(mrg8g_set_state(g, st), 0);
    set_word(1);
    calls(MRG8G_ERR_TIMEOUT);
    EXPECT(mrg8g_get_state(g, after), 0);
    EXPECT(std::memcmp(st, after, sizeof(st)), 0);
    mrg8g_request r{};
    r.generator = MRG8G_NO_GENERATOR;
    r.seed = 7;
    r.n = 1000;
    r.kind = MRG8G_F64_SHIFTED;
    uint64_t ticket = 0;
    EXPECT(mrg8g_server_submit(sv, &r, &ticket), 0);
    mrg8g_completion c{};
    uint32_t count = 0;
    for (int i = 0; i < 100 && !count; ++i) EXPECT(mrg8g_server_poll(sv, &c, 1, &count, 100000), 0);
    EXPECT(count, 1);
    EXPECT(c.status, MRG8G_ERR_TIMEOUT);
    EXPECT(mrg8g_server_read(sv, ticket, host.data(), 8), MRG8G_ERR_TIMEOUT);
    EXPECT(mrg8g_server_submit(sv, &r, &ticket), MRG8G_ERR_TIMEOUT);
    EXPECT(mrg8g_server_destroy(sv), 0);
    set_word(0);
    calls(0);
    EXPECT(mrg8g_batch_destroy(b), 0);
    EXPECT(mrg8g_destroy(g), 0);
    return bad;
}

int main(int argc, char** argv) {
    if (argc == 2 && !std::strcmp(argv[1], "host")) check_host();
    else return 2;
    EXPECT(cudaDeviceSynchronize(), 0);
    std::printf("bad=%d\n", bad);
    return bad != 0;
}
