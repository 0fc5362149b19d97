// short_waits.cu -- the tensor-core kernels built a second time, in a namespace of
// their own, with waits that give up after one short look.
#define MRG8G_WAIT_LIMIT_NS 1
#define MRG8G_LOOK_NS 1000
#define mrg8g mrg8g_short
#include "mrg8g_tables.cpp"
#include "mrg8g_tensor.cu"
#undef mrg8g

// `args`: mrg8g::TensorArgs or BatchArgs, the same struct in either namespace.
extern "C" int short_setup() {
    cudaError_t e = mrg8g_short::upload_tables_tensor();
    if (e == cudaSuccess) e = mrg8g_short::prepare_tensor();
    return (int)e;
}
extern "C" int short_tensor(const void* args, int sms) {
    return (int)mrg8g_short::launch_tensor(*static_cast<const mrg8g_short::TensorArgs*>(args), sms, nullptr);
}
extern "C" int short_batch(const void* args, int kind, int sms) {
    return (int)mrg8g_short::launch_tensor_batch(*static_cast<const mrg8g_short::BatchArgs*>(args), kind, sms, nullptr);
}
