// The buffer pool of the host layer (vesper_b200/host/src/tensor.cpp) against a fake CUDA runtime: no device is needed, and a stream is
// busy, being captured or idle as a test says.  Which buffer a stream gets is what is checked.
#include "fake_cuda.h"

#include <thread>

using namespace vesper;

#define CHECK(x) do { if (!(x)) { std::printf("FAIL %s:%d: %s\n", __FILE__, __LINE__, #x); return 1; } } while (0)

namespace {
cudaStream_t raw(const Stream& s) { return static_cast<cudaStream_t>(s.raw_handle()); }
// a buffer of n floats made and let go of with `s` current
void* use(Stream& s, int64_t n) {
    Stream::set_current(s);
    return empty({n}, DType::Float32, Device::CUDA).data_ptr<char>();
}
}  // namespace

int main() {
    Stream a(Device::CUDA), b(Device::CUDA);
    Stream& legacy = Stream::default_stream(Device::CUDA);

    // a stream gets its own buffer again at once; another stream not while the first has work queued
    fake::streams[raw(a)] = fake::kBusy;
    void* p = use(a, 1000);
    CHECK(use(a, 1000) == p);
    CHECK(use(b, 1000) != p);
    CHECK(cudaGetLastError() == cudaSuccess);
    // the same from another thread
    void* q = nullptr;
    std::thread([&] { q = use(b, 1000); }).join();
    CHECK(q != p);
    // a stream that is being captured is neither idle nor may be asked
    fake::streams[raw(a)] = fake::kCapturing;
    void* c = use(a, 5000);
    CHECK(use(b, 5000) != c);
    use(a, 5000);                                             // its own or a new one, without a question to b
    // idle: anyone's
    fake::streams[raw(a)] = fake::kIdle;
    CHECK(use(b, 1000) == p || use(b, 1000) == q);
    const size_t before = fake::blocks.size();
    use(b, 1000); use(a, 1000);
    CHECK(fake::blocks.size() == before);

    // made on one stream, let go of on another: no third stream's while either is busy
    Stream d(Device::CUDA);
    {
        Stream::set_current(a);
        Tensor t = empty({70000}, DType::Float32, Device::CUDA);
        p = t.data_ptr<char>();
        Stream::set_current(b);
    }
    fake::streams[raw(a)] = fake::streams[raw(b)] = fake::kBusy;
    CHECK(use(d, 70000) != p);
    CHECK(use(b, 70000) != p);
    fake::streams[raw(a)] = fake::kIdle;
    CHECK(use(d, 70000) != p);
    fake::streams[raw(b)] = fake::kIdle;

    // the default stream's work is in order with that of every stream: it gets a busy stream's buffer, but a third stream does not get it from there
    Stream e(Device::CUDA);
    fake::streams[raw(e)] = fake::kBusy;
    p = use(e, 300000);
    CHECK(use(legacy, 300000) == p);
    CHECK(use(d, 300000) != p);

    // a destroyed stream's handle does not pass for a new stream's
    {
        Stream f(Device::CUDA);
        fake::streams[raw(f)] = fake::kBusy;
        p = use(f, 900000);
    }
    Stream g(Device::CUDA);
    CHECK(use(g, 900000) != p);
    std::puts("OK");
    return 0;
}
