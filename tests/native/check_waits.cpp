// check_waits.cpp -- what a wait that gave up inside a kernel leads to, with the
// library's own objects linked in.
//
//   check_waits host
//       The device's error word is set, as such a kernel does: every call that
//       launches or waits returns MRG8G_ERR_TIMEOUT and leaves handles as they
//       were, and all work again once the word is cleared.
//   check_waits kernel
//       The kernels with waits that give up after one short look (short_waits.cu),
//       against set-up and steps that take microseconds: a wait gives up
//       somewhere in at least a quarter of the launches.  Each launch ends without
//       a CUDA error, its outputs are complete if the word is not set, and the
//       library's own next launch is complete.
#include <cuda_runtime.h>

#include <cstdio>
#include <cstring>
#include <vector>

#include "mrg8g.h"
#include "mrg8g_internal.h"
#include "mrg8g_runtime.h"

extern "C" int short_setup();
extern "C" int short_tensor(const void* args, int sms);
extern "C" int short_batch(const void* args, int kind, int sms);

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

constexpr int kTries = 12;
static int launches = 0, ended = 0;

static uint32_t word() {
    uint32_t v = 0;
    EXPECT(cudaMemcpy(&v, mrg8g::device_fault(), sizeof(v), cudaMemcpyDefault), 0);
    return v;
}

// The library's launch, launches that give up, and the library's again; `launch` is
// told whether to give up.
template <class L>
static void check_launches(uint64_t bytes, const void* d, L&& launch) {
    std::vector<char> want(bytes), got(bytes);
    const auto run = [&](bool give_up, char* to) {
        set_word(0);
        EXPECT(cudaMemset((void*)d, 0x5A, bytes), 0);
        EXPECT(launch(give_up), 0);
        EXPECT(cudaDeviceSynchronize(), 0);
        EXPECT(cudaMemcpy(to, d, bytes, cudaMemcpyDeviceToHost), 0);
        return word();
    };
    EXPECT(run(false, want.data()), 0);
    for (int i = 0; i < kTries; ++i) {
        const uint32_t gave_up = run(true, got.data());
        ++launches;
        ended += gave_up;
        if (!gave_up) EXPECT(std::memcmp(want.data(), got.data(), bytes), 0);
    }
    EXPECT(run(false, got.data()), 0);
    EXPECT(std::memcmp(want.data(), got.data(), bytes), 0);
}

static int check_kernel() {
    using namespace mrg8g;
    const int sms = device_sms();
    EXPECT(short_setup(), 0);
    char* d = nullptr;
    EXPECT(cudaMalloc(&d, 32 << 20), 0);
    uint32_t st[8];
    EXPECT(mrg8g_seed_state(11, st), 0);
    const uint64_t sizes[] = {1000, 40000, 3000001};
    for (int kind = MRG8G_U32; kind <= MRG8G_F32_SHIFTED; ++kind)
        for (uint64_t n : sizes)
            check_launches(n * kind_elem_bytes(kind), d, [&](bool give_up) -> int {
                TensorArgs a{};
                std::memcpy(a.st, st, sizeof(st));
                a.n = n;
                a.quarters = (n + kTcQuarter - 1) / kTcQuarter;
                a.out = d;
                a.kind = kind;
                a.fault = device_fault();
                return give_up ? short_tensor(&a, sms) : (int)launch_tensor(a, sms, nullptr);
            });
    // Batches of one kind and of all, in tiles of 64 rows.
    constexpr uint32_t kCount = 5, kTile = 64 * 32 * kBatchLayoutV;
    BatchInst* d_insts = nullptr;
    uint32_t *d_base = nullptr, *d_counter = nullptr;
    EXPECT(cudaMalloc(&d_insts, kCount * sizeof(BatchInst)), 0);
    EXPECT(cudaMalloc(&d_base, (kCount + 1) * sizeof(uint32_t)), 0);
    EXPECT(cudaMalloc(&d_counter, sizeof(uint32_t)), 0);
    for (int kind = -1; kind <= MRG8G_F32_SHIFTED; ++kind)
        for (uint64_t n : {1000ull, 600000ull}) {
            BatchInst in[kCount]{};
            uint32_t base[kCount + 1];
            for (uint32_t i = 0; i < kCount; ++i) {
                std::memcpy(in[i].st, st, sizeof(st));
                in[i].offset = 1000003ull * i;
                in[i].n = n;
                in[i].out = d + 8 * n * i;
                in[i].kind = kind < 0 ? (int)i : kind;
            }
            const uint32_t tiles = (uint32_t)tile_prefix(in, kCount, kTile, base);
            EXPECT(cudaMemcpy(d_insts, in, sizeof(in), cudaMemcpyHostToDevice), 0);
            EXPECT(cudaMemcpy(d_base, base, sizeof(base), cudaMemcpyHostToDevice), 0);
            check_launches(8 * n * kCount, d, [&](bool give_up) -> int {
                EXPECT(cudaMemset(d_counter, 0, sizeof(uint32_t)), 0);
                BatchArgs a{};
                a.insts = d_insts;
                a.tile_base = d_base;
                a.ninst = kCount;
                a.tile_elems = kTile;
                a.ntiles = tiles;
                a.counter = d_counter;
                a.fault = device_fault();
                return give_up ? short_batch(&a, kind, sms) : (int)launch_tensor_batch(a, kind, sms, nullptr);
            });
        }
    std::printf("%d of %d launches gave up\n", ended, launches);
    EXPECT(4 * ended >= launches, true);
    return bad;
}

int main(int argc, char** argv) {
    if (argc == 2 && !std::strcmp(argv[1], "host")) check_host();
    else if (argc == 2 && !std::strcmp(argv[1], "kernel")) check_kernel();
    else return 2;
    EXPECT(cudaDeviceSynchronize(), 0);
    std::printf("bad=%d\n", bad);
    return bad != 0;
}
