// A CUDA runtime that computes nothing, for programs that compile vesper_b200/host/src/tensor.cpp in: streams are busy, being captured or idle, and the
// device status word holds, what a test says.
#pragma once

#include <vesper/core/tensor.h>
#include <vesper_b200.h>

#include <cuda_runtime.h>

#include <cstdio>
#include <cstdlib>
#include <map>
#include <set>

namespace fake {
enum State { kIdle, kBusy, kCapturing };
std::map<cudaStream_t, State> streams;
std::map<void*, size_t> blocks;         // what the driver has given out, at most `memory` bytes
size_t memory = size_t{180} << 30;
size_t given() { size_t n = 0; for (auto& b : blocks) n += b.second; return n; }
cudaError_t last = cudaSuccess;
int32_t status = 0;             // the device's status word
char detail[64];
}  // namespace fake

extern "C" {
const char* cudaGetErrorString(cudaError_t) { return "fake"; }
cudaError_t cudaGetLastError() { cudaError_t e = fake::last; fake::last = cudaSuccess; return e; }
cudaError_t cudaGetDevice(int* d) { *d = 0; return cudaSuccess; }
cudaError_t cudaMalloc(void** p, size_t n) {
    static uintptr_t next = 1 << 20;
    if (fake::given() + n > fake::memory) return fake::last = cudaErrorMemoryAllocation;
    *p = reinterpret_cast<void*>(next);
    next += 1 << 20;
    fake::blocks[*p] = n;
    return cudaSuccess;
}
cudaError_t cudaFree(void* p) { fake::blocks.erase(p); return cudaSuccess; }
cudaError_t cudaStreamCreate(cudaStream_t* s) {
    *s = static_cast<cudaStream_t>(std::malloc(1));
    fake::streams[*s] = fake::kIdle;
    return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t s) { fake::streams.erase(s); std::free(s); return cudaSuccess; }      // the address may come again
cudaError_t cudaStreamSynchronize(cudaStream_t s) { if (s) fake::streams.at(s) = fake::kIdle; return cudaSuccess; }
cudaError_t cudaStreamIsCapturing(cudaStream_t s, cudaStreamCaptureStatus* c) {
    *c = fake::streams.at(s) == fake::kCapturing ? cudaStreamCaptureStatusActive : cudaStreamCaptureStatusNone;
    return cudaSuccess;
}
cudaError_t cudaStreamQuery(cudaStream_t s) {
    const auto current = static_cast<cudaStream_t>(vesper::Stream::current(vesper::Device::CUDA).raw_handle());
    if (fake::streams.at(s) == fake::kCapturing || (current && fake::streams.at(current) == fake::kCapturing)) {
        std::puts("FAIL: a stream was queried that captures, or by a thread that does");
        std::exit(1);
    }
    return fake::last = fake::streams.at(s) == fake::kBusy ? cudaErrorNotReady : cudaSuccess;
}
cudaError_t cudaMemcpy(void*, const void*, size_t, cudaMemcpyKind) { return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void*, const void*, size_t, cudaMemcpyKind, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaMemsetAsync(void*, int, size_t, cudaStream_t) { return cudaSuccess; }
const char* vb200_strerror(int) { return ""; }
const char* vb200_last_error_detail(void) { return fake::detail; }
int vb200_kernel_status_on_host(int, const volatile int32_t** word) { *word = &fake::status; return VB200_OK; }
int vb200_kernel_status_of(int32_t word) {
    std::snprintf(fake::detail, sizeof(fake::detail), "code %d, site 0x%x", word >> 24, word & 0xFFFFFF);
    return word == 0 ? VB200_OK : word >> 24 == 2 ? VB200_ERR_CACHE_OVERFLOW : VB200_ERR_KERNEL_TIMEOUT;
}
int vb200_check_kernel_status(int, void*) { const int rc = vb200_kernel_status_of(fake::status); fake::status = 0; return rc; }
int vb200_kv_append(int, void*, int32_t, int32_t, int32_t, int32_t, int32_t, int32_t, const vb200_tensor4*, const vb200_tensor4*, const vb200_tensor4*, const vb200_tensor4*, int32_t,
                    const vb200_rope*) { return 0; }
}
