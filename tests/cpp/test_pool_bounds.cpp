// What the host layer's buffer pool keeps (vesper_b200/host/src/tensor.cpp), against a fake CUDA runtime.
#include "fake_cuda.h"

#include <vector>

using namespace vesper;

#define CHECK(x) do { if (!(x)) { std::printf("FAIL %s:%d: %s\n", __FILE__, __LINE__, #x); return 1; } } while (0)

namespace {
constexpr size_t kGiB = size_t{1} << 30;
Tensor buffer(size_t bytes) { return empty({static_cast<int64_t>(bytes / 4)}, DType::Float32, Device::CUDA); }
}  // namespace

int main() {
    Stream a(Device::CUDA);
    Stream::set_current(a);
    // a gigabyte and a little: less than an eighth more, and used again
    buffer(kGiB + 4096);
    CHECK(fake::given() <= kGiB + kGiB / 8 + kGiB / 16);
    const size_t one = fake::given();
    buffer(kGiB + 8192);
    CHECK(fake::given() == one);
    // the free blocks of many large buffers go back beyond 32 GiB
    {
        std::vector<Tensor> t;
        for (int i = 0; i < 40; ++i) t.push_back(buffer(kGiB + kGiB / 2));
        CHECK(fake::given() >= 60 * kGiB);
    }
    CHECK(fake::given() <= 32 * kGiB);
    // not those that a stream still works on, and none while the thread captures
    for (const auto state : {fake::kBusy, fake::kCapturing}) {
        {
            std::vector<Tensor> t;
            for (int i = 0; i < 30; ++i) t.push_back(buffer(kGiB + kGiB / 2));
            fake::streams[static_cast<cudaStream_t>(a.raw_handle())] = state;
        }
        CHECK(fake::given() >= 45 * kGiB);
        fake::streams[static_cast<cudaStream_t>(a.raw_handle())] = fake::kIdle;
        buffer(1024);
        CHECK(fake::given() <= 32 * kGiB);
    }
    // a full device: what is free goes back and the buffer is had after all
    fake::memory = 10 * kGiB;
    Tensor large = buffer(9 * kGiB);
    CHECK(large.data_ptr<char>() != nullptr && cudaGetLastError() == cudaSuccess);
    bool refused = false;
    try { buffer(4 * kGiB); } catch (const std::runtime_error&) { refused = true; }
    CHECK(refused);
    std::puts("OK");
    return 0;
}
