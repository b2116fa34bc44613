// A set device status word becomes an exception where the host layer waits for the device (vesper_b200/host/src/tensor.cpp), against a fake CUDA runtime.
#include "fake_cuda.h"

#include <string>

using namespace vesper;

#define CHECK(x) do { if (!(x)) { std::printf("FAIL %s:%d: %s\n", __FILE__, __LINE__, #x); return 1; } } while (0)

namespace {
template <typename F>
std::string error_of(F f) {
    try { f(); } catch (const std::runtime_error& e) { return e.what(); }
    return "";
}
}  // namespace

int main() {
    Stream s(Device::CUDA);
    Tensor t = empty({4}, DType::Float32, Device::CUDA);
    float out[4];
    auto read = [&] { t.copy_to_host(out); };
    auto wait = [&] { s.synchronize(); };
    CHECK(error_of(read).empty() && error_of(wait).empty());
    for (const int code : {1, 3}) {
        fake::status = code << 24 | 0x43;
        CHECK(error_of(read).find("site 0x43") != std::string::npos);        // names the wait
        CHECK(error_of(read).empty());                                       // and was cleared by that
        fake::status = code << 24 | 0x52;
        CHECK(error_of(wait).find("site 0x52") != std::string::npos);
        CHECK(error_of(wait).empty());
    }
    fake::status = 2 << 24 | 7;                                              // a full sequence: left to vb200_check_kernel_status
    CHECK(error_of(read).empty() && error_of(wait).empty() && fake::status == (2 << 24 | 7));
    Stream::default_stream(Device::CPU).synchronize();
    std::puts("OK");
    return 0;
}
