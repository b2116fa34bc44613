// fp32 attention forward on CUDA cores (fp32 in, fp32 math, fp32 out): head dims other than 64 and 128, short sequences, and calls without the workspace
// that the tensor-core kernel (attention_f32_sm100.cu) needs.
//
// This is the dtype the reference's flash op runs in
// (flash_attention_cuda_dispatch, src/ops/cuda/flash_attention.cu:518-544), so
// it keeps full fp32 accuracy instead of down-converting to a tensor-core
// type.  Same math as flash_attention_cpu_dispatch
// (src/ops/flash_attention.cpp:218-364): s = scale * q.k, causal j <= i,
// online softmax, O = acc / l, LSE = m + ln l.
//
// Tiling: 64 query rows x 64 keys per step, 128 or 256 threads, products as in f32_tiles.cuh (packed fp32 FMAs, 8 x 4 and 8 x 8
// register blocks, or half as many rows).  A CTA keeps one K and one V tile: V arrives while the scores are computed, the next K tile during the
// softmax and the value product, so both loads hide behind arithmetic without a second buffer, and two CTAs
// share an SM, or three (head_dim 64 with 128 threads: 16 x 2048 x 64 360 us against 364 with two, 64 x 1024 x 16 226 against 233, although
// 84 bytes spill).  A row's 64 weights are written and read by the same half warp.
#include "f32_tiles.cuh"
#include "kernels.h"
#include "hybrid.cuh"

namespace vb200 {

namespace {

using namespace f32t;

constexpr int kPitchP = kTile + 4;     // weights: rows ty and ty + 1 of one warp in distinct banks

__device__ __forceinline__ float rowgroup_max(float v) {
#pragma unroll
    for (int o = 8; o >= 1; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xFFFFFFFFu, v, o));
    return v;
}
__device__ __forceinline__ float rowgroup_sum(float v) {
#pragma unroll
    for (int o = 8; o >= 1; o >>= 1) v += __shfl_xor_sync(0xFFFFFFFFu, v, o);
    return v;
}

template <int DMAX> constexpr int smem_floats() { return 3 * kTile * DMAX + kTile * kPitchP; }

// R query rows per thread
template <int DMAX, int R>
__global__ void __launch_bounds__(1024 / R, R == 8 && DMAX == 64 ? 3 : 2) prefill_f32_kernel(PrefillParams p) {
    extern __shared__ __align__(16) float smem[];
    constexpr int G = DMAX / 64, kThreads = 1024 / R, kStep = kTile / R;
    float* Qs = smem;
    float* Ks = Qs + kTile * DMAX;
    float* Vs = Ks + kTile * DMAX;
    float* Ps = Vs + kTile * DMAX;

    const int D = p.D, tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
    const int qt = gridDim.x - 1 - blockIdx.x;   // longest (last) causal tiles first
    const int hq = blockIdx.y, b = blockIdx.z;
    const int hkv = hq / (p.Hq / p.Hkv);
    const int q0 = qt * kTile, words = D >> 2;

    const float* qg = static_cast<const float*>(p.q.ptr) + b * p.q.sb + hq * p.q.sh;
    const float* kg = static_cast<const float*>(p.k.ptr) + b * p.k.sb + hkv * p.k.sh;
    const float* vg = static_cast<const float*>(p.v.ptr) + b * p.v.sb + hkv * p.v.sh;

    int kv_end = p.Skv;
    if (p.causal) kv_end = min(p.Skv, p.start_pos + min(q0 + kTile, p.T));
    // the first tiles of Q (unless it is rotated on the way in), K and V are on their way at once
    if (p.q_rope_table == nullptr) load_rows<DMAX, Swizzle::A>(Qs, qg, p.q.ss, q0, p.T, D, tid, kThreads);
    load_rows<DMAX, Swizzle::B>(Ks, kg, p.k.ss, 0, kv_end, D, tid, kThreads);
    cp_async_commit();
    load_rows<DMAX, Swizzle::None>(Vs, vg, p.v.ss, 0, kv_end, D, tid, kThreads);
    cp_async_commit();

    for (int i = p.q_rope_table != nullptr ? tid : kTile * (DMAX / 4); i < kTile * (DMAX / 4); i += kThreads) {
        const int r = i / (DMAX / 4), c = i % (DMAX / 4);
        float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
        if (q0 + r < p.T && c < words) {
            x = *reinterpret_cast<const float4*>(qg + static_cast<long long>(q0 + r) * p.q.ss + c * 4);
            const float2* tp = p.q_rope_table + static_cast<long long>(q0 + r) * (D / 2) + c * 2;
            float2 cs0 = tp[0], cs1 = tp[1];
            float t1 = __fmul_rn(x.x, cs0.x), t2 = __fmul_rn(x.y, cs0.y), t3 = __fmul_rn(x.x, cs0.y), t4 = __fmul_rn(x.y, cs0.x);
            x.x = __fsub_rn(t1, t2); x.y = __fadd_rn(t3, t4);
            t1 = __fmul_rn(x.z, cs1.x); t2 = __fmul_rn(x.w, cs1.y); t3 = __fmul_rn(x.z, cs1.y); t4 = __fmul_rn(x.w, cs1.x);
            x.z = __fsub_rn(t1, t2); x.w = __fadd_rn(t3, t4);
        }
        *reinterpret_cast<float4*>(Qs + r * DMAX + 4 * (c ^ swz_a(r))) = x;
    }

    float m_i[R], l_i[R];
    Pair acc[R][2 * G];
#pragma unroll
    for (int i = 0; i < R; ++i) {
        m_i[i] = -INFINITY; l_i[i] = 0.f;
#pragma unroll
        for (int g = 0; g < 2 * G; ++g) acc[i][g] = 0;
    }

    for (int k0 = 0; k0 < kv_end; k0 += kTile) {
        if (k0 == 0) cp_async_wait_but_last(); else cp_async_wait_all();
        __syncthreads();   // K has arrived (and Q, the first time); the previous V tile is fully consumed
        if (k0 > 0) {
            load_rows<DMAX, Swizzle::None>(Vs, vg, p.v.ss, k0, kv_end, D, tid, kThreads);
            cp_async_commit();
        }

        float s[R][4];
        tile_abt<DMAX, R>(s, Qs, Ks, words, tx, ty);

        cp_async_wait_all();
        __syncthreads();   // V has arrived; K is fully consumed
        if (k0 + kTile < kv_end) {
            load_rows<DMAX, Swizzle::B>(Ks, kg, p.k.ss, k0 + kTile, kv_end, D, tid, kThreads);
            cp_async_commit();
        }

        // keys past the end, or past a row's own position: only the last tiles have any
        const bool edge = k0 + kTile > p.Skv || (p.causal && k0 + kTile - 1 > p.start_pos + q0);
#pragma unroll
        for (int i = 0; i < R; ++i) {
            const int row = q0 + ty + kStep * i;
#pragma unroll
            for (int j = 0; j < 4; ++j) s[i][j] *= p.scale;
            if (edge) {
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const int kc = k0 + 4 * tx + j;
                    if (!(kc < p.Skv && (!p.causal || kc <= p.start_pos + row))) s[i][j] = -INFINITY;
                }
            }
            const float mx = rowgroup_max(fmaxf(fmaxf(s[i][0], s[i][1]), fmaxf(s[i][2], s[i][3])));
            const float m_new = fmaxf(m_i[i], mx);
            const float m_use = (m_new == -INFINITY) ? 0.f : m_new;
            const float alpha = expf(m_i[i] - m_use);       // exp(-inf) = 0 on the first tile
            float4 w;
            w.x = expf(s[i][0] - m_use); w.y = expf(s[i][1] - m_use); w.z = expf(s[i][2] - m_use); w.w = expf(s[i][3] - m_use);
            *reinterpret_cast<float4*>(Ps + (ty + kStep * i) * kPitchP + 4 * tx) = w;
            l_i[i] = l_i[i] * alpha + ((w.x + w.y) + (w.z + w.w));      // per-thread partial; reduced at the end
            m_i[i] = m_new;
            const Pair a2 = dup2(alpha);
#pragma unroll
            for (int g = 0; g < 2 * G; ++g) mul2(acc[i][g], a2);
        }
        __syncwarp();
        tile_ab<DMAX, kPitchP, G, false, R>(acc, Ps, Vs, 0, min(kTile, kv_end - k0), 0, tx, ty);      // (weights and rows past the keys are zero)
    }

    float* og = static_cast<float*>(p.o.ptr) + b * p.o.sb + hq * p.o.sh;
#pragma unroll
    for (int i = 0; i < R; ++i) {
        const int row = q0 + ty + kStep * i;
        const float l = rowgroup_sum(l_i[i]);
        if (row >= p.T) continue;
        const float inv = 1.0f / l;
#pragma unroll
        for (int g = 0; g < G; ++g) {
            const int dc = g * 64 + tx * 4;
            if (dc < D) {
                const float4 x = quad4(acc[i][2 * g], acc[i][2 * g + 1]);
                *reinterpret_cast<float4*>(og + static_cast<long long>(row) * p.o.ss + dc) = make_float4(x.x * inv, x.y * inv, x.z * inv, x.w * inv);
            }
        }
        if (p.lse && tx == 0)
            p.lse[(static_cast<long long>(b) * p.Hq + hq) * p.T + row] = m_i[i] + logf(l);
    }
}

template <int DMAX, int R>
int launch_t(cudaStream_t s, const PrefillParams& p, bool alone = false) {
    constexpr int kSmem = smem_floats<DMAX>() * static_cast<int>(sizeof(float)), kAlone = 116 * 1024;      // two of kAlone do not fit an SM
    const int smem = alone ? kAlone : kSmem;
    static thread_local bool configured[64] = {};      // per device ordinal: the attribute belongs to the device's context
    int dev = 0;
    VB200_CUDA_TRY(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64) return set_detail(VB200_ERR_NO_DEVICE, "device ordinal out of range");
    if (!configured[dev]) {
        VB200_CUDA_TRY(cudaFuncSetAttribute(prefill_f32_kernel<DMAX, R>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem > kAlone ? kSmem : kAlone));
        configured[dev] = true;
    }
    dim3 grid((p.T + kTile - 1) / kTile, p.Hq, p.B);
    prefill_f32_kernel<DMAX, R><<<grid, 1024 / R, smem, s>>>(p);
    note_launch();
    note_prefill_kernel("prefill_f32_kernel");
    VB200_CUDA_TRY(cudaPeekAtLastError());
    return VB200_OK;
}

}  // namespace

// The tensor cores (attention_f32_sm100.cu) from the second block of 64 keys on, and for short portions of many heads, whose 128-row tiles are mostly
// padding, from 512 keys on.  This kernel / those: 16 heads, 512 x 64 50 / 21 us; 16, 2048 x 128 671 / 97; 1024, 128 x 128 199 / 154; 64 heads, 65 x 64
// 14.7 / 12.9, but 64 x 64 10.5 / 10.8 and 1024 heads, 64 x 64 45 / 65; 16 new rows of 1024 heads behind 240 keys 125 / 132, 496 238 / 223, of 128 heads
// behind 112 16.7 / 14.7.
bool prefill_f32_on_tensor_cores(int D, int T, int keys, int heads) {
    return (D == 64 || D == 128) && keys > 64 && (T > 64 || heads <= 128 || keys >= 512);
}

int launch_prefill_f32(cudaStream_t s, const PrefillParams& p) {
    if (p.D % 4 != 0 || p.D > 128 || p.D < 4) return set_detail(VB200_ERR_UNSUPPORTED, "fp32 attention needs head_dim % 4 == 0 and <= 128");
    // Query rows per thread: 4 (256 threads) while the grid leaves SMs with few CTAs or the sequences are short, where a tile's latency counts; 8 (128 threads),
    // which read shared memory less, for long grids.  4 / 8 rows: one head, 64 x 32 7.7 / 10.4 us; 8 heads, 512 x 64 48.8 / 52.2; 16 heads, 1400 x 64 (352 CTAs)
    // 201 / 262; 1024 heads, 64 x 32 35.4 / 37.4; but 128 heads, 256 x 64 (512 CTAs) 63.7 / 59.3; 4 heads, 8192 x 64 1598 / 1346.
    const long long ctas = static_cast<long long>((p.T + kTile - 1) / kTile) * p.Hq * p.B;
    const bool few = ctas <= 3 * device_sm_count() || p.Skv <= 2 * kTile;
    if (p.split != nullptr) return launch_prefill_f32_sm100(s, p, p.split);
    if (p.D <= 64) return few ? launch_t<64, 4>(s, p) : launch_t<64, 8>(s, p);
    // head_dim above 64, long causal grids of one to two CTAs per SM: the row tiles with the most keys are the call's length, and an SM to itself each shortens them
    // more than a second CTA hides.  Two / one per SM: 2 heads, 8192 x 128 1861 / 1155 us; 6 heads, 2048 447 / 329; 32 heads, 512 133 / 125; 16 heads, 1024 232 / 232;
    // but 128 heads, 128 38 / 44.
    const bool alone = p.causal && p.Skv >= 512 && ctas > device_sm_count() && ctas <= 2 * device_sm_count();
    return few ? launch_t<128, 4>(s, p, alone) : launch_t<128, 8>(s, p);
}

}  // namespace vb200
