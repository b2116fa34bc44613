// The fp32 operator on a device with no room for the terms of its operands (vesper_b200/host/src/attention.cpp), against a fake CUDA runtime: it runs with what a
// call cannot do without, and does not fail where it needed no such memory before.
#include "fake_cuda.h"

#include <vesper/ops/flash_attention.h>

#include <vector>

namespace fake {
size_t all = size_t{1} << 30, least = 0, passed = 0;
bool called = false;
}  // namespace fake

extern "C" {
size_t vb200_prefill_workspace_bytes(const vb200_prefill_args*) { return fake::all; }
size_t vb200_prefill_workspace_bytes_min(const vb200_prefill_args*) { return fake::least; }
int vb200_prefill_fwd(const vb200_prefill_args* a) { fake::called = true; fake::passed = a->workspace_bytes; return VB200_OK; }
size_t vb200_attention_bwd_workspace_bytes(const vb200_attention_bwd_args*) { return fake::all; }
size_t vb200_attention_bwd_workspace_bytes_min(const vb200_attention_bwd_args* a) { return sizeof(float) * a->B * a->H * a->N; }
int vb200_attention_bwd(const vb200_attention_bwd_args* a) { fake::called = true; fake::passed = a->workspace_bytes; return VB200_OK; }
int vb200_apply_rope(int, void*, float*, const float*, const float*, int32_t, int32_t, int32_t, int32_t) { return VB200_OK; }
size_t vb200_decode_workspace_bytes(const vb200_decode_args*) { return 0; }
int vb200_decode_fwd(const vb200_decode_args*) { return VB200_OK; }
int vb200_repeat_kv(int, void*, int32_t, const vb200_tensor4*, void*, int32_t, int32_t, int32_t, int32_t, int32_t) { return VB200_OK; }
void vb200_rope_inv_freq(float, int32_t, float*) {}
}

using namespace vesper;

#define CHECK(x) do { if (!(x)) { std::printf("FAIL %s:%d: %s\n", __FILE__, __LINE__, #x); return 1; } } while (0)

int main() {
    const std::vector<int64_t> shape{1, 2, 1000, 64};
    Tensor t = empty(shape, DType::Float32, Device::CUDA), lse = empty({1, 2, 1000}, DType::Float32, Device::CUDA);
    for (const bool full : {false, true}) {
        if (full) fake::memory = fake::given() + (size_t{16} << 20);
        fake::called = false;
        ops::flash_attention(t, t, t, 0.125f);
        CHECK(fake::called && (full ? fake::passed < fake::all : fake::passed >= fake::all));
        fake::called = false;
        ops::flash_attention_backward(t, t, t, t, t, lse, 0.125f);
        CHECK(fake::called && (full ? fake::passed >= 8000 && fake::passed < fake::all : fake::passed >= fake::all));
        CHECK(cudaGetLastError() == cudaSuccess);
        fake::all *= 2;          // (a block of the first size is free now)
    }
    std::puts("OK");
    return 0;
}
