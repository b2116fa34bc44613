// y = x W^T for bf16 activations x[M,K] and bf16 weights W[N,K] (the layout of the reference's
// nn::Linear::weight, src/nn/linear.cpp:19, whose forward is matmul(input, weight.transpose(0,1)),
// src/nn/linear.cpp:41-48) on the sm_100a tensor cores, fp32 accumulation in TMEM.
//
// Three kernels share the TMA / tcgen05 plumbing:
//   linear_pair_kernel    M > 64 (prompt processing).  Persistent pairs of CTAs walk 256 x 256 output tiles;
//                         x rows are the UMMA M operand, W rows the N operand; TMA ring,
//                         two TMEM accumulators so the epilogue of one tile overlaps the next mainloop.
//   linear_wide_kernel    the same with single CTAs and 128 x 256 tiles: grouped rows, and few rows
//                         beyond a multiple of 256.
//   linear_skinny_kernel  M <= 64 (one token per sequence).  The product is weight-bandwidth bound,
//                         so the roles swap: 128 W rows are the UMMA M operand and the (zero padded)
//                         16, 32 or 64 token rows the N operand; K is split over the CTAs of a thread-block
//                         cluster, which scatter their partial tiles through distributed shared
//                         memory; each CTA sums and finishes its tokens in a fixed order (deterministic).
// Epilogues (fused, per output element): store bf16 | store fp32 | fp32 accumulate into the residual
// stream (optionally plus a second fp32 addend) | squared ReLU -> bf16 | SwiGLU over interleaved (gate, up) weight rows -> bf16 (src/nn/swiglu.cpp:36-48,
// ops::silu_mul src/ops/elementwise.cpp:1297-1328) | the same with max(gate, 0).
#include "cluster_pair.cuh"
#include "kernels.h"

#include <cuda.h>
#include <cstdio>

namespace vb200 {
namespace {

constexpr int kBK = 64;                 // K elements per stage = one 128-byte swizzle row
constexpr int kTileA = 128;             // rows of the UMMA M operand
constexpr int kThreads = 192;           // warp 0: TMA producer, warp 1: MMA issuer, warps 2-5: epilogue
constexpr int kABytes = kTileA * kBK * 2;

struct LinearMaps {
    CUtensorMap a;   // UMMA M operand rows
    CUtensorMap b;   // UMMA N operand rows
};

__device__ __forceinline__ void tma_load_2d(void* smem_dst, const CUtensorMap* m, uint64_t* bar, int c0, int c1) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes"
        " [%0], [%1, {%3, %4}], [%2];"
        : : "r"(smem_u32(smem_dst)), "l"(reinterpret_cast<uint64_t>(m)), "r"(smem_u32(bar)), "r"(c0), "r"(c1)
        : "memory");
}
// 32-byte global accesses (sm_100): half as many store instructions per row segment as 16-byte ones.  The
// interface promises 16-byte alignment only, so a segment that is not 32-byte aligned goes as two halves.
__device__ __forceinline__ void st_global_v8(void* ptr, const uint32_t (&w)[8]) {
    if ((reinterpret_cast<uintptr_t>(ptr) & 31) == 0) {
        asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};"
                     ::"l"(ptr), "r"(w[0]), "r"(w[1]), "r"(w[2]), "r"(w[3]), "r"(w[4]), "r"(w[5]), "r"(w[6]), "r"(w[7]) : "memory");
    } else {
        uint4* p4 = static_cast<uint4*>(ptr);
        p4[0] = make_uint4(w[0], w[1], w[2], w[3]);
        p4[1] = make_uint4(w[4], w[5], w[6], w[7]);
    }
}
__device__ __forceinline__ void ld_global_v8(const void* ptr, uint32_t (&w)[8]) {
    if ((reinterpret_cast<uintptr_t>(ptr) & 31) == 0) {
        asm volatile("ld.global.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                     : "=r"(w[0]), "=r"(w[1]), "=r"(w[2]), "=r"(w[3]), "=r"(w[4]), "=r"(w[5]), "=r"(w[6]), "=r"(w[7]) : "l"(ptr) : "memory");
    } else {
        const uint4* p4 = static_cast<const uint4*>(ptr);
        const uint4 a = p4[0], b = p4[1];
        w[0] = a.x; w[1] = a.y; w[2] = a.z; w[3] = a.w; w[4] = b.x; w[5] = b.y; w[6] = b.z; w[7] = b.w;
    }
}
__device__ __forceinline__ float silu_f(float g) { return g / (1.0f + __expf(-g)); }
template <int EPI> constexpr bool kGated = EPI == VB200_EPI_SWIGLU || EPI == VB200_EPI_REGLU;
// the gate's activation of a gated epilogue
template <int EPI> __device__ __forceinline__ float gate_f(float g) { return EPI == VB200_EPI_REGLU ? fmaxf(g, 0.f) : silu_f(g); }

// The residual values that 32 consecutive columns of one row are added to; loaded ahead of the product they wait for.
__device__ __forceinline__ void load_row32(const LinearParams& p, int row, int col0, uint32_t (&was)[32]) {
    const float* out = static_cast<const float*>(p.out) + static_cast<long long>(row) * p.ldo + col0;
    if (col0 + 32 <= p.N) {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            uint32_t w[8];
            ld_global_v8(out + 8 * j, w);
#pragma unroll
            for (int e = 0; e < 8; ++e) was[8 * j + e] = w[e];
        }
    } else {
#pragma unroll
        for (int j = 0; j < 32; ++j) was[j] = col0 + j < p.N ? __float_as_uint(out[j]) : 0u;
    }
}

// One output element group of the tiled kernels: 32 consecutive columns of one row; `was`: their residual values (+= epilogue).
template <int EPI>
__device__ __forceinline__ void store_row32(const LinearParams& p, int row, int col0, uint32_t (&acc)[32], const uint32_t (&was)[32]) {
    if (p.row_scale != nullptr) {                // deferred RMSNorm: this row's 1/rms
        const float rs = __ldg(p.row_scale + row);
#pragma unroll
        for (int j = 0; j < 32; ++j) acc[j] = __float_as_uint(__uint_as_float(acc[j]) * rs);
    }
    if (p.bias != nullptr) {                     // nn::Linear's bias (src/nn/linear.cpp:44-46)
#pragma unroll
        for (int j = 0; j < 32; ++j)
            if (col0 + j < p.N) acc[j] = __float_as_uint(__uint_as_float(acc[j]) + __ldg(p.bias + col0 + j));
    }
    if (kGated<EPI>) {
        // columns (2j, 2j+1) = (gate_j, up_j) -> out[row, col0/2 + j]
        __nv_bfloat16* out = static_cast<__nv_bfloat16*>(p.out) + static_cast<long long>(row) * p.ldo + (col0 >> 1);
        const int n_out = min(16, (p.N - col0) >> 1);
        uint32_t packed[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            float a0 = gate_f<EPI>(__uint_as_float(acc[4 * j])) * __uint_as_float(acc[4 * j + 1]);
            float a1 = gate_f<EPI>(__uint_as_float(acc[4 * j + 2])) * __uint_as_float(acc[4 * j + 3]);
            packed[j] = Elem<__nv_bfloat16>::pack2(a0, a1);
        }
        if (n_out == 16) {
            st_global_v8(out, packed);
        } else {
#pragma unroll
            for (int j = 0; j < 16; ++j) {
                if (j >= n_out) break;
                const uint32_t u = packed[j >> 1];
                reinterpret_cast<uint16_t*>(out)[j] = static_cast<uint16_t>((j & 1) ? (u >> 16) : (u & 0xFFFF));
            }
        }
        return;
    }
    const int n_valid = min(32, p.N - col0);
    if (EPI == VB200_EPI_RELU2) {
#pragma unroll
        for (int j = 0; j < 32; ++j) { const float r = fmaxf(__uint_as_float(acc[j]), 0.f); acc[j] = __float_as_uint(r * r); }
    }
    if (EPI == VB200_EPI_ADD_F32 && p.addend != nullptr) {
        const float* ad = p.addend + static_cast<long long>(row) * p.ldo + col0;
#pragma unroll
        for (int j = 0; j < 32; ++j)
            if (j < n_valid) acc[j] = __float_as_uint(__uint_as_float(acc[j]) + ad[j]);
    }
    if (EPI == VB200_EPI_BF16 || EPI == VB200_EPI_RELU2) {
        __nv_bfloat16* out = static_cast<__nv_bfloat16*>(p.out) + static_cast<long long>(row) * p.ldo + col0;
        if (n_valid == 32) {
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                uint32_t w8[8];
#pragma unroll
                for (int e = 0; e < 8; ++e) w8[e] = Elem<__nv_bfloat16>::pack2(__uint_as_float(acc[16 * j + 2 * e]), __uint_as_float(acc[16 * j + 2 * e + 1]));
                st_global_v8(out + 16 * j, w8);
            }
        } else {
#pragma unroll
            for (int j = 0; j < 32; ++j)
                if (j < n_valid) out[j] = __float2bfloat16_rn(__uint_as_float(acc[j]));
        }
    } else {
        float* out = static_cast<float*>(p.out) + static_cast<long long>(row) * p.ldo + col0;
        if (n_valid == 32) {
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                uint32_t w8[8];
#pragma unroll
                for (int e = 0; e < 8; ++e) {
                    float v = __uint_as_float(acc[8 * j + e]);
                    if (EPI == VB200_EPI_ADD_F32) v += __uint_as_float(was[8 * j + e]);
                    w8[e] = __float_as_uint(v);
                    acc[8 * j + e] = w8[e];                     // the new residual value, for the scaled copy below
                }
                st_global_v8(out + 8 * j, w8);
            }
        } else {
#pragma unroll
            for (int j = 0; j < 32; ++j) {
                if (j >= n_valid) break;
                float v = __uint_as_float(acc[j]);
                if (EPI == VB200_EPI_ADD_F32) v += __uint_as_float(was[j]);
                out[j] = v;
                acc[j] = __float_as_uint(v);
            }
        }
        if (EPI == VB200_EPI_ADD_F32 && p.scaled_copy != nullptr) {
            __nv_bfloat16* cp = static_cast<__nv_bfloat16*>(p.scaled_copy) + static_cast<long long>(row) * p.N + col0;
            if (n_valid == 32) {
                const float4* g4 = reinterpret_cast<const float4*>(p.copy_scale + col0);
#pragma unroll
                for (int j = 0; j < 2; ++j) {
                    uint32_t w8[8];
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        const float4 gw = __ldg(g4 + 4 * j + e);
                        w8[2 * e] = Elem<__nv_bfloat16>::pack2(__uint_as_float(acc[16 * j + 4 * e]) * gw.x, __uint_as_float(acc[16 * j + 4 * e + 1]) * gw.y);
                        w8[2 * e + 1] = Elem<__nv_bfloat16>::pack2(__uint_as_float(acc[16 * j + 4 * e + 2]) * gw.z, __uint_as_float(acc[16 * j + 4 * e + 3]) * gw.w);
                    }
                    st_global_v8(cp + 16 * j, w8);
                }
            } else {
#pragma unroll
                for (int j = 0; j < 32; ++j)
                    if (j < n_valid) cp[j] = __float2bfloat16_rn(__uint_as_float(acc[j]) * __ldg(p.copy_scale + col0 + j));
            }
        }
    }
}

// ------------------------------------------------------------------------------------------------
// Wide kernel: out[m, n] = sum_k x[m,k] W[n,k], tiles of 128 rows (m) x BN columns (n).
// ------------------------------------------------------------------------------------------------
template <int BN>
struct WideCfg {
    static constexpr int kStages = 4;
    static constexpr int kBBytes = BN * kBK * 2;
    static constexpr int kStageBytes = kABytes + kBBytes;
    static constexpr int kBarOffset = kStages * kStageBytes;
    static constexpr int kSmemBytes = kBarOffset + 256 + 1024;      // barriers + slack for 1024-byte alignment
    static constexpr int kTmemCols = 2 * BN;                        // two accumulators
    static_assert(kTmemCols <= 512 && (kTmemCols & (kTmemCols - 1)) == 0, "TMEM allocation is a power of two <= 512");
};

// GROUPED: rows sorted by group, each group with weights of its own; the row tiles come from a device list.
template <int BN, int EPI, bool GROUPED = false>
__global__ void __launch_bounds__(kThreads, 1)
linear_wide_kernel(const __grid_constant__ LinearMaps maps, LinearParams p) {
    using C = WideCfg<BN>;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
    uint64_t* full = reinterpret_cast<uint64_t*>(smem + C::kBarOffset);
    uint64_t* empty = full + C::kStages;
    uint64_t* acc_full = empty + C::kStages;      // [2]
    uint64_t* acc_empty = acc_full + 2;           // [2]
    uint64_t* drain = acc_empty + 2;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(drain + 1);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
    int* row_tiles = reinterpret_cast<int*>(tmem_slot + 2);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    int m_tiles = (p.M + kTileA - 1) / kTileA;
    const int n_tiles = (p.N + BN - 1) / BN;
    const int k_blocks = (p.K + kBK - 1) / kBK;
    const WaitCtx ctx{abort_flag, p.status};

    if (threadIdx.x == 0) {
        *abort_flag = 0;
        for (int i = 0; i < C::kStages; ++i) { mbar_init(&full[i], 1); mbar_init(&empty[i], 1); }
        for (int i = 0; i < 2; ++i) { mbar_init(&acc_full[i], 1); mbar_init(&acc_empty[i], 4); }
        mbar_init(drain, 1);
        mbar_fence_init();
        tma_prefetch_desc(&maps.a);
        tma_prefetch_desc(&maps.b);
    }
    if (warp == 1) { tmem_alloc(tmem_slot, C::kTmemCols); tmem_relinquish(); }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    // the next kernel in the stream may be scheduled now (it waits for this grid to finish before it reads
    // anything); the activations may come from the kernel launched just before this one
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    if (GROUPED) {                                // read once: copies, products and epilogue must agree on the number of tiles, or each waits for the others
        if (threadIdx.x == 0) *row_tiles = max(0, min(__ldcg(p.group_tile_count), p.group_tile_max));
        __syncthreads();
        m_tiles = *row_tiles;
    }
    const int tiles = m_tiles * n_tiles;

    if (warp == 0) {
        if (lane == 0) {
            uint32_t it = 0;
            for (int t = blockIdx.x; t < tiles && !*abort_flag; t += gridDim.x) {
                // consecutive CTAs share a W tile through L2; grouped: a row tile, and a group's W stays in L2 for its few row tiles
                const int mt = GROUPED ? t / n_tiles : t % m_tiles, nt = GROUPED ? t % n_tiles : t / m_tiles;
                int row0 = mt * kTileA, w0 = nt * BN;
                if (GROUPED) { const int4 g = __ldcg(p.group_tiles + mt); row0 = g.x; w0 += g.z * p.group_rows; }
                for (int kb = 0; kb < k_blocks; ++kb, ++it) {
                    const int s = it % C::kStages;
                    if (it >= C::kStages && !mbar_wait(&empty[s], ((it / C::kStages) - 1) & 1, ctx, 0x41)) break;
                    uint8_t* st = smem + s * C::kStageBytes;
                    mbar_arrive_expect_tx(&full[s], C::kStageBytes);
                    tma_load_2d(st, &maps.a, &full[s], kb * kBK, row0);
                    tma_load_2d(st + kABytes, &maps.b, &full[s], kb * kBK, w0);
                }
            }
        }
    } else if (warp == 1) {
        constexpr uint32_t idesc = make_idesc_f16(1, 0, 0, kTileA, BN);
        const bool leader = elect_one();              // (the whole warp walks: see the note at umma_ss)
        const uint32_t tmem = uniform(tmem_base);
        uint32_t it = 0, tile_no = 0;
        bool ok = true;
        for (int t = blockIdx.x; t < tiles && ok; t += gridDim.x, ++tile_no) {
            const int buf = tile_no & 1;
            if (tile_no >= 2) ok = mbar_wait_warp(&acc_empty[buf], ((tile_no >> 1) - 1) & 1, ctx, 0x42);
            if (!ok) break;
            tc_fence_after();
            for (int kb = 0; kb < k_blocks; ++kb, ++it) {
                const int s = it % C::kStages;
                if (!mbar_wait_warp(&full[s], (it / C::kStages) & 1, ctx, 0x43)) { ok = false; break; }
                tc_fence_after();
                const uint32_t a_addr = smem_u32(smem + s * C::kStageBytes);
                const uint64_t ad = make_smem_desc_sw128(a_addr, 16, 1024), bd = make_smem_desc_sw128(a_addr + kABytes, 16, 1024);
                if (leader) {
#pragma unroll
                    for (int kk = 0; kk < kBK / 16; ++kk)          // 32 bytes further, in the descriptors' units of 16
                        umma_ss(tmem + buf * BN, ad + 2 * kk, bd + 2 * kk, idesc, (kb | kk) ? 1u : 0u);
                    umma_commit(&empty[s]);           // the stage is free once these MMAs have read it
                }
            }
            if (ok && leader) umma_commit(&acc_full[buf]);
        }
        // drain: no MMA may be in flight when TMEM is freed (also on the abort path)
        if (leader) umma_commit(drain);
        mbar_wait_warp(drain, 0, ctx, 0x44);
    } else {
        const int quarter = warp & 3;                 // TMEM lanes this warp may read
        uint32_t tile_no = 0;
        for (int t = blockIdx.x; t < tiles; t += gridDim.x, ++tile_no) {
            const int mt = GROUPED ? t / n_tiles : t % m_tiles, nt = GROUPED ? t % n_tiles : t / m_tiles;
            const int buf = tile_no & 1;
            if (!mbar_wait_warp(&acc_full[buf], (tile_no >> 1) & 1, ctx, 0x45)) break;
            tc_fence_after();
            int row = mt * kTileA, row_end = p.M;
            if (GROUPED) { const int4 g = __ldcg(p.group_tiles + mt); row = g.x; row_end = g.y; }
            row += quarter * 32 + lane;
#pragma unroll 1
            for (int c = 0; c < BN / 32; ++c) {
                uint32_t acc[32], was[32];
                const int col0 = nt * BN + c * 32;
                if (EPI == VB200_EPI_ADD_F32 && row < row_end && col0 < p.N) load_row32(p, row, col0, was);
                tmem_ld32(tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) + buf * BN + c * 32, acc);
                tmem_ld_wait();
                if (row < row_end && col0 < p.N) store_row32<EPI>(p, row, col0, acc, was);
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&acc_empty[buf]);
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) tmem_dealloc(tmem_base, C::kTmemCols);
    abort_linger(abort_flag);
}

// ------------------------------------------------------------------------------------------------
// Pair kernel: out[m, n] = sum_k x[m,k] W[n,k] on tiles of 256 rows x BN columns, each by a cluster of two CTAs (cta_group::2).
//
// With every SM at work single CTAs wait for L2: a 128 x 256 tile reads 48 KB per 64-column K block, 148 of them 16 TB/s at
// the rate they reached (0.45 us per block; 0.33 us with few SMs at work).  A pair reads 64 KB for twice the product: each CTA
// loads its 128 rows of x and half of the tile's rows of W, and the tensor cores read W's halves from both.  Eight epilogue warps have
// two chunks of the residual on their way.  4096 rows, single CTAs -> pairs: 3072 x 2048 53.4 -> 37.3 us (1380 TFLOP/s), 8448 x 2048
// 151 -> 98 (1440), 2048 x 2048 onto the residual 52 -> 36, 2048 x 5632 95 -> 78, 11264 x 2048 gated 143 -> 131; 3003 rows, 2048 x 8448 128 -> 95.
// ------------------------------------------------------------------------------------------------
constexpr int kPairEpilogue = 8;                    // epilogue warps: each 32 rows x half of a tile's columns
constexpr int kPairThreads = 64 + 32 * kPairEpilogue;
struct PairMaps { CUtensorMap a, b, b_half; };      // x; W in boxes of half a tile's columns, and of a quarter's
template <int BN>
struct PairCfg {
    static constexpr int kBBytes = BN / 2 * kBK * 2;
    static constexpr int kStageBytes = kABytes + kBBytes;
    static constexpr int kStages = BN == 256 ? 6 : 8;
    static constexpr int kBarOffset = kStages * kStageBytes;
    static constexpr int kSmemBytes = kBarOffset + 256 + 1024;
    static constexpr int kTmemCols = 2 * BN;                        // two accumulators
    static_assert(kTmemCols <= 512 && (kTmemCols & (kTmemCols - 1)) == 0, "TMEM allocation is a power of two <= 512");
    static_assert((2 * kStages + 5) * 8 + 8 <= 256, "barriers");
};

// TMA load whose completion bytes go to a barrier that may live in the peer CTA (shared::cluster address); no multicast
__device__ __forceinline__ void tma_load_2d_pair(void* smem_dst, const CUtensorMap* m, uint32_t bar_cluster_addr, int c0, int c1) {
    asm volatile(
        "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.tile.mbarrier::complete_tx::bytes"
        " [%0], [%1, {%3, %4}], [%2];"
        : : "r"(smem_u32(smem_dst)), "l"(reinterpret_cast<uint64_t>(m)), "r"(bar_cluster_addr), "r"(c0), "r"(c1)
        : "memory");
}

// What a pair computes at a time: a tile, or (from tile `whole` on) half of its columns.
struct PairUnit { int row_tile, col0; bool half; };
template <int BN>
__device__ __forceinline__ PairUnit pair_unit(int u, int whole, int m_tiles) {
    const bool half = u >= whole;
    const int t = half ? whole + (u - whole) / 2 : u;
    return PairUnit{t % m_tiles, t / m_tiles * BN + (half ? ((u - whole) & 1) * (BN / 2) : 0), half};      // consecutive pairs share a W tile through L2
}

template <int BN, int EPI>
__global__ void __launch_bounds__(kPairThreads, 1)
linear_pair_kernel(const __grid_constant__ PairMaps maps, LinearParams p, int whole) {
    using C = PairCfg<BN>;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
    uint64_t* full = reinterpret_cast<uint64_t*>(smem + C::kBarOffset);       // the leader's: both CTAs' loads of a stage
    uint64_t* empty = full + C::kStages;
    uint64_t* acc_full = empty + C::kStages;      // [2]
    uint64_t* acc_empty = acc_full + 2;           // [2], the leader's: both CTAs' epilogue warps
    uint64_t* drain = acc_empty + 2;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(drain + 1);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int cta = static_cast<int>(cluster_ctarank()), pairs = gridDim.x / 2;
    const int m_tiles = (p.M + 2 * kTileA - 1) / (2 * kTileA), units = 2 * (m_tiles * ((p.N + BN - 1) / BN)) - whole;
    const int k_blocks = (p.K + kBK - 1) / kBK;
    const WaitCtx ctx{abort_flag, p.status};

    if (threadIdx.x == 0) {
        *abort_flag = 0;
        for (int i = 0; i < C::kStages; ++i) { mbar_init(&full[i], 1); mbar_init(&empty[i], 1); }
        for (int i = 0; i < 2; ++i) { mbar_init(&acc_full[i], 1); mbar_init(&acc_empty[i], 2 * kPairEpilogue); }
        mbar_init(drain, 1);
        mbar_fence_init();
        tma_prefetch_desc(&maps.a);
        tma_prefetch_desc(&maps.b);
    }
    if (warp == 1) { tmem_alloc2(tmem_slot, C::kTmemCols); tmem_relinquish2(); }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    cluster_arrive();
    cluster_wait();                               // both CTAs' barriers exist before anything crosses the pair
    const uint32_t tmem_base = *tmem_slot;
    // the next kernel in the stream may be scheduled now (it waits for this grid to finish before it reads
    // anything); the activations may come from the kernel launched just before this one
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");

    if (warp == 0) {
        if (lane == 0) {
            uint32_t it = 0;
            for (int u = blockIdx.x / 2; u < units && !*abort_flag; u += pairs) {
                const PairUnit w = pair_unit<BN>(u, whole, m_tiles);
                const int row0 = (w.row_tile * 2 + cta) * kTileA, cols = w.half ? BN / 4 : BN / 2, w0 = w.col0 + cta * cols;
                const CUtensorMap* mb = w.half ? &maps.b_half : &maps.b;
                for (int kb = 0; kb < k_blocks; ++kb, ++it) {
                    const int s = it % C::kStages;
                    if (it >= C::kStages && !mbar_wait(&empty[s], ((it / C::kStages) - 1) & 1, ctx, 0x61)) break;
                    uint8_t* st = smem + s * C::kStageBytes;
                    if (cta == 0) mbar_arrive_expect_tx(&full[s], 2 * (kABytes + cols * kBK * 2));
                    const uint32_t bar = map_to_cta(smem_u32(&full[s]), 0);
                    tma_load_2d_pair(st, &maps.a, bar, kb * kBK, row0);
                    tma_load_2d_pair(st + kABytes, mb, bar, kb * kBK, w0);
                }
            }
        }
    } else if (warp == 1) {
        if (cta == 0) {
            const bool leader = elect_one();
            const uint32_t tmem = uniform(tmem_base);
            uint32_t it = 0, tile_no = 0;
            bool ok = true;
            for (int u = blockIdx.x / 2; u < units && ok; u += pairs, ++tile_no) {
                const uint32_t idesc = u < whole ? make_idesc_f16(1, 0, 0, 2 * kTileA, BN) : make_idesc_f16(1, 0, 0, 2 * kTileA, BN / 2);
                const int buf = tile_no & 1;
                if (tile_no >= 2) ok = mbar_wait_warp(&acc_empty[buf], ((tile_no >> 1) - 1) & 1, ctx, 0x62);
                if (!ok) break;
                tc_fence_after();
                for (int kb = 0; kb < k_blocks; ++kb, ++it) {
                    const int s = it % C::kStages;
                    if (!mbar_wait_warp(&full[s], (it / C::kStages) & 1, ctx, 0x63)) { ok = false; break; }
                    tc_fence_after();
                    const uint32_t a_addr = smem_u32(smem + s * C::kStageBytes);
                    const uint64_t ad = make_smem_desc_sw128(a_addr, 16, 1024), bd = make_smem_desc_sw128(a_addr + kABytes, 16, 1024);
                    if (leader) {
#pragma unroll
                        for (int kk = 0; kk < kBK / 16; ++kk)
                            umma2_ss(tmem + buf * BN, ad + 2 * kk, bd + 2 * kk, idesc, (kb | kk) ? 1u : 0u);
                        umma2_commit(&empty[s]);      // the stage is free in both CTAs once these MMAs have read it
                    }
                }
                if (ok && leader) umma2_commit(&acc_full[buf]);
            }
            if (leader) umma2_commit(drain);              // behind every MMA above (also after a break)
        }
        __syncwarp();
    } else {
        const int quarter = warp & 3;                 // TMEM lanes this warp may read
        uint32_t tile_no = 0;
        for (int u = blockIdx.x / 2; u < units; u += pairs, ++tile_no) {
            const int buf = tile_no & 1;
            const PairUnit w = pair_unit<BN>(u, whole, m_tiles);
            const int chunks = BN / (kPairEpilogue / 4) / 32 / (w.half ? 2 : 1), col_first = (warp - 2) / 4 * chunks * 32;
            const int row = (w.row_tile * 2 + cta) * kTileA + quarter * 32 + lane, col_tile = w.col0 + col_first;
            uint32_t was[2][32];                      // residual values: two chunks on their way before they are needed
            auto ahead = [&](int c) {
                if (EPI == VB200_EPI_ADD_F32 && c < chunks && row < p.M && col_tile + c * 32 < p.N) load_row32(p, row, col_tile + c * 32, was[c & 1]);
            };
            ahead(0);
            ahead(1);
            if (!mbar_wait_warp(&acc_full[buf], (tile_no >> 1) & 1, ctx, 0x65)) break;
            tc_fence_after();
#pragma unroll
            for (int c = 0; c < BN / (kPairEpilogue / 4) / 32; ++c) {
                if (c == chunks) break;
                uint32_t acc[32];
                tmem_ld32(tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) + buf * BN + col_first + c * 32, acc);
                tmem_ld_wait();
                if (c + 1 == chunks) {                // the accumulator is in registers: the next product may have its columns
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive_cluster(map_to_cta(smem_u32(&acc_empty[buf]), 0));
                }
                const int col0 = col_tile + c * 32;
                if (row < p.M && col0 < p.N) store_row32<EPI>(p, row, col0, acc, was[c & 1]);
                ahead(c + 2);
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    // No MMA may be in flight when TMEM is freed, also on the abort path.  Waited for behind the epilogue, by both CTAs: the limit of a wait
    // covers the last products, not the whole walk over the tiles.
    if (threadIdx.x == 32) mbar_wait(drain, 0, ctx, 0x64);
    __syncwarp();
    cluster_arrive();
    cluster_wait();                                   // nobody signals the peer or reads its tiles any more
    if (warp == 1) tmem_dealloc2(tmem_base, C::kTmemCols);
    abort_linger(abort_flag);
}

// ------------------------------------------------------------------------------------------------
// Skinny kernel: out[m, n] = sum_k x[m,k] W[n,k] for m < MT <= 64.  One CTA = 128 W rows x one K slice;
// the `splits` CTAs of a cluster hold the K slices of the same 128 rows.
//
// What bounds it: the weights' bytes, and, in a chain of such products (a decode step), the time from the predecessor's end to
// its own.  So the ring's first weight tiles are loaded before the predecessor has finished (two CTAs fit an SM), and the cluster's
// sum is scattered: CTA r finishes tokens [r, r + 1) * share of the 128 rows, every other CTA stores its partials of them straight
// into r's shared memory (st.async, counted by a barrier of r), and r adds them in rank order (bit-reproducible) while it already
// holds the residual rows that they go onto.  Dependent products of 8 tokens, one leading CTA's sum behind two cluster
// barriers -> now: 2048 x 2048 8.2 -> 4.4 us, 2048 x 5632 10.6 -> 7.7, 11264 x 2048 14.2 -> 12.0, 160 x 4096 5.7 -> 5.2; 32000 x
// 2048, one slice, 22.4 -> 22.6.
// ------------------------------------------------------------------------------------------------
// stores of V values to another CTA's shared memory, counted by the barrier `bar` there (both shared::cluster addresses)
template <int V>
__device__ __forceinline__ void st_async(uint32_t addr, const float* v, uint32_t bar) {
    if (V == 4)
        asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v4.f32 [%0], {%1, %2, %3, %4}, [%5];"
                     ::"r"(addr), "f"(v[0]), "f"(v[1]), "f"(v[2]), "f"(v[3]), "r"(bar) : "memory");
    else if (V == 2)
        asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v2.f32 [%0], {%1, %2}, [%3];" ::"r"(addr), "f"(v[0]), "f"(v[1]), "r"(bar) : "memory");
    else
        asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.f32 [%0], %1, [%2];" ::"r"(addr), "f"(v[0]), "r"(bar) : "memory");
}
template <int V>
__device__ __forceinline__ void load_v(float (&v)[V], const float* p) {
    if (V == 4) { const float4 t = *reinterpret_cast<const float4*>(p); v[0] = t.x; v[V > 1 ? 1 : 0] = t.y; v[V > 2 ? 2 : 0] = t.z; v[V > 3 ? 3 : 0] = t.w; }
    else if (V == 2) { const float2 t = *reinterpret_cast<const float2*>(p); v[0] = t.x; v[V > 1 ? 1 : 0] = t.y; }
    else v[0] = *p;
}

template <int MT>
struct SkinnyCfg {
    static constexpr int kResident = 2;                                   // CTAs per SM that registers and shared memory are laid out for
    static constexpr int kStages = MT == 16 ? 5 : MT == 32 ? 4 : 3;      // as many as leave room for them
    static constexpr int kBBytes = MT * kBK * 2;
    static constexpr int kStageBytes = kABytes + kBBytes;
    static constexpr int kMaxSplits = MT == 64 ? 5 : 8;
    static constexpr int kRedOffset = kStages * kStageBytes;              // partials of the other CTAs [splits - 1][128][share] fp32
    static constexpr int kRedTokens = MT == 16 ? 24 : MT == 32 ? 48 : 64; // the largest (splits - 1) * share: 7 CTAs, with 64 tokens 5
    static constexpr int kBarOffset = kRedOffset + kRedTokens * kTileA * 4;
    static constexpr int kSmemBytes = kBarOffset + 256 + 1024;
    static constexpr int kTmemCols = MT < 32 ? 32 : MT;
    static_assert(kResident * (kSmemBytes + MT * 4 + 1024) <= 228 * 1024, "shared memory of the CTAs of an SM");
};

// The cluster's sum: CTA r adds the partials of tokens [r * share, (r + 1) * share) in rank order.  V = 4, or share where that is smaller: tokens
// per remote store.  (A pair of CTAs exchanges one store of a lane in about three cycles, whatever its width: single values cost 0.2 us per token.)
template <int MT, int V>
__device__ __forceinline__ void cluster_sum(float (&acc)[MT], float* red, float* self, uint64_t* red_full, int rank, int splits, int share, int m_count, int own,
                                            int row, const WaitCtx& ctx) {
    const uint32_t there = smem_u32(red) + row * share * 4, bar = smem_u32(red_full);
#pragma unroll
    for (int j = 0; j < MT; j += V) {
        if (j >= m_count) break;
        const int dst = j / share, at = j - dst * share;
        if (dst == rank) {
#pragma unroll
            for (int e = 0; e < V; ++e) self[row * share + at + e] = acc[j + e];
        } else {
            const int slot = rank < dst ? rank : rank - 1;
            st_async<V>(map_to_cta(there + (slot * kTileA * share + at) * 4, dst), &acc[j], map_to_cta(bar, dst));
        }
    }
    if (own == 0) return;
    mbar_wait_warp<true>(red_full, 0, ctx, 0x54);
#pragma unroll
    for (int j = 0; j < (MT / 2 < V ? V : MT / 2); j += V) {
        if (j >= own) break;
        float sum[V];
#pragma unroll
        for (int e = 0; e < V; ++e) sum[e] = 0.f;
        for (int r = 0; r < splits; ++r) {               // fixed order: bit-reproducible
            float v[V];
            load_v<V>(v, (r == rank ? self : red + (r < rank ? r : r - 1) * kTileA * share) + row * share + j);
#pragma unroll
            for (int e = 0; e < V; ++e) sum[e] = r == 0 ? v[e] : sum[e] + v[e];
        }
#pragma unroll
        for (int e = 0; e < V; ++e) acc[j + e] = sum[e];
    }
}

template <int MT, int EPI>
__global__ void __launch_bounds__(kThreads, SkinnyCfg<MT>::kResident)
linear_skinny_kernel(const __grid_constant__ LinearMaps maps, LinearParams p, int splits) {
    using C = SkinnyCfg<MT>;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
    uint64_t* full = reinterpret_cast<uint64_t*>(smem + C::kBarOffset);
    uint64_t* empty = full + C::kStages;
    uint64_t* acc_full = empty + C::kStages;
    uint64_t* red_full = acc_full + 1;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(red_full + 1);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int rank = splits > 1 ? static_cast<int>(cluster_ctarank()) : 0;
    const int nt = blockIdx.x / splits;
    const int k_blocks = (p.K + kBK - 1) / kBK;
    const int kb_per = (k_blocks + splits - 1) / splits;
    const int kb0 = rank * kb_per;
    const int nkb = max(0, min(k_blocks, kb0 + kb_per) - kb0);
    const int m_count = min(p.M, MT);
    int share = (m_count + splits - 1) / splits;                     // tokens that a CTA of the cluster finishes: 1, 2 or a multiple of 4
    if (splits > 1 && share > 2) share = (share + 3) & ~3;
    const int tok0 = rank * share, own = max(0, min(m_count - tok0, share));
    const WaitCtx ctx{abort_flag, p.status};
    __shared__ float s_inv_rms[MT];

    if (threadIdx.x == 0) {
        *abort_flag = 0;
        for (int i = 0; i < C::kStages; ++i) { mbar_init(&full[i], 1); mbar_init(&empty[i], 1); }
        mbar_init(acc_full, 1);
        mbar_init(red_full, 1);
        mbar_fence_init();
        const int wide = min(share, 4);
        mbar_arrive_expect_tx(red_full, splits > 1 ? static_cast<uint32_t>((splits - 1) * ((own + wide - 1) / wide * wide) * kTileA * 4) : 0u);
        tma_prefetch_desc(&maps.a);
        tma_prefetch_desc(&maps.b);
    }
    if (warp == 1) { tmem_alloc(tmem_slot, C::kTmemCols); tmem_relinquish(); }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    if (splits > 1) cluster_arrive();             // this CTA's barriers exist; waited for before the first remote store
    // Programmatic dependent launch: the next kernel of the stream may be scheduled as soon as every CTA of
    // this grid is here, and this grid was scheduled while its predecessor was still running.  Weights do
    // not depend on the predecessor, so their first ring of TMA loads goes out BEFORE griddepcontrol.wait
    // and streams while the predecessor finishes; only the activation loads and the epilogue's global
    // accesses wait for it.  (Fetching the rest of the slice into L2 as well made dependent products slower.)
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");

    float acc[MT];
#pragma unroll
    for (int j = 0; j < MT; ++j) acc[j] = 0.0f;
    const int n = nt * kTileA + (warp & 3) * 32 + lane;              // the epilogue thread's W row
    constexpr int kHeld = EPI == VB200_EPI_ADD_F32 ? 16 : 1;
    // residual values of 16 of the CTA's own tokens at a time: 32 would take 178 registers, and only one CTA would fit an SM (33 rows on 3-stage rings, one CTA -> two:
    // 4096 x 4096 23.6 -> 11.9 us, 2048 x 5632 17.4 -> 11.7, 8192 x 8192 38.1 -> 27.0; with one CTA and 6 stages they had been 27.7, 20.5, 62.7)
    float held[kHeld];
    auto load_held = [&](int j0) {
#pragma unroll
        for (int j = 0; j < kHeld; ++j)
            if (j0 + j < own) held[j] = __ldcg(static_cast<const float*>(p.out) + static_cast<long long>(tok0 + j0 + j) * p.ldo + n);
    };
    float gain = 0.f;

    if (warp == 0) {
        if (lane == 0) {
            const int pre = min(nkb, C::kStages);
            for (int i = 0; i < pre; ++i) {
                mbar_arrive_expect_tx(&full[i], C::kStageBytes);
                tma_load_2d(smem + i * C::kStageBytes, &maps.a, &full[i], (kb0 + i) * kBK, nt * kTileA);     // 128 W rows
            }
            asm volatile("griddepcontrol.wait;" ::: "memory");
            for (int i = 0; i < pre; ++i)
                tma_load_2d(smem + i * C::kStageBytes + kABytes, &maps.b, &full[i], (kb0 + i) * kBK, 0);      // the token rows (zero filled past M)
            for (int i = pre; i < nkb; ++i) {
                const int s = i % C::kStages;
                if (!mbar_wait(&empty[s], ((i / C::kStages) - 1) & 1, ctx, 0x51)) break;
                uint8_t* st = smem + s * C::kStageBytes;
                mbar_arrive_expect_tx(&full[s], C::kStageBytes);
                tma_load_2d(st, &maps.a, &full[s], (kb0 + i) * kBK, nt * kTileA);
                tma_load_2d(st + kABytes, &maps.b, &full[s], (kb0 + i) * kBK, 0);
            }
        }
        __syncwarp();
        if (splits > 1) cluster_wait();
    } else if (warp == 1) {
        {
            constexpr uint32_t idesc = make_idesc_f16(1, 0, 0, kTileA, MT);
            const bool leader = elect_one();
            const uint32_t tmem = uniform(tmem_base);
            for (int i = 0; i < nkb; ++i) {
                const int s = i % C::kStages;
                if (!mbar_wait_warp(&full[s], (i / C::kStages) & 1, ctx, 0x52)) break;
                tc_fence_after();
                const uint32_t a_addr = smem_u32(smem + s * C::kStageBytes);
                const uint64_t ad = make_smem_desc_sw128(a_addr, 16, 1024), bd = make_smem_desc_sw128(a_addr + kABytes, 16, 1024);
                if (leader) {
#pragma unroll
                    for (int kk = 0; kk < kBK / 16; ++kk) umma_ss(tmem, ad + 2 * kk, bd + 2 * kk, idesc, (i | kk) ? 1u : 0u);
                    umma_commit(&empty[s]);
                }
            }
            if (leader) umma_commit(acc_full);       // completes once every MMA above has finished (also after a break)
        }
        __syncwarp();
        if (splits > 1) cluster_wait();
    } else {
        const int quarter = warp & 3;
        if (splits > 1) cluster_wait();
        asm volatile("griddepcontrol.wait;" ::: "memory");      // before any global access of the epilogue
        if (EPI == VB200_EPI_ADD_F32 && n < p.N) {
            load_held(0);
            if (p.scaled_copy != nullptr) gain = __ldg(p.copy_scale + n);
        }
        if (p.rms_rows != nullptr) {
            // deferred RMSNorm: 1/rms of the CTA's own token rows, computed while the weights stream (these warps are idle
            // until the accumulator is complete); one warp per row, every load of a 2048-column chunk in flight
            const int nv = p.rms_dim / 4;
            for (int j = warp - 2; j < own; j += 4) {
                const float4* hr = reinterpret_cast<const float4*>(p.rms_rows + static_cast<long long>(tok0 + j) * p.rms_ld);
                float ss = 0.f;
                for (int c0 = 0; c0 < nv; c0 += 512) {
                    float4 v[16];
#pragma unroll
                    for (int i = 0; i < 16; ++i) {
                        const int c = c0 + lane + 32 * i;
                        v[i] = c < nv ? __ldcg(hr + c) : make_float4(0.f, 0.f, 0.f, 0.f);
                    }
#pragma unroll
                    for (int i = 0; i < 16; ++i) ss += v[i].x * v[i].x + v[i].y * v[i].y + v[i].z * v[i].z + v[i].w * v[i].w;
                }
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xFFFFFFFFu, ss, o);
                if (lane == 0) s_inv_rms[j] = 1.0f / sqrtf(ss / static_cast<float>(p.rms_dim) + p.rms_eps);
            }
        }
        // wait even when this slice is empty: the commit above always arrives
        if (mbar_wait_warp(acc_full, 0, ctx, 0x53) && nkb > 0) {
            tc_fence_after();
#pragma unroll
            for (int c = 0; c < MT / 16; ++c) {
                uint32_t r[16];
                tmem_ld16(tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) + c * 16, r);
                tmem_ld_wait();
#pragma unroll
                for (int j = 0; j < 16; ++j) acc[c * 16 + j] = __uint_as_float(r[j]);
            }
        }
        tc_fence_before();

        if (splits > 1) {
            const int row = quarter * 32 + lane;
            float* red = reinterpret_cast<float*>(smem + C::kRedOffset);
            float* self = reinterpret_cast<float*>(smem);       // this CTA's own partials, where its ring was: every product has read it
            if (share >= 4) cluster_sum<MT, 4>(acc, red, self, red_full, rank, splits, share, m_count, own, row, ctx);
            else if (share == 2) cluster_sum<MT, 2>(acc, red, self, red_full, rank, splits, share, m_count, own, row, ctx);
            else cluster_sum<MT, 1>(acc, red, self, red_full, rank, splits, share, m_count, own, row, ctx);
        }

        if (p.rms_rows != nullptr) {
            asm volatile("bar.sync 2, 128;" ::: "memory");       // s_inv_rms written by the four epilogue warps
#pragma unroll
            for (int j = 0; j < MT; ++j) acc[j] *= (j < own ? s_inv_rms[j] : 0.f);
        }
        if (p.bias != nullptr && n < p.N) {
            const float bv = __ldg(p.bias + n);
#pragma unroll
            for (int j = 0; j < MT; ++j) acc[j] += bv;
        }
        if (kGated<EPI>) {
            __nv_bfloat16* out = static_cast<__nv_bfloat16*>(p.out);
#pragma unroll
            for (int j = 0; j < MT; ++j) {
                if (j >= own) break;
                const float other = __shfl_xor_sync(0xFFFFFFFFu, acc[j], 1);     // odd lanes hold the `up` rows
                if (!(lane & 1) && n + 1 < p.N)
                    out[static_cast<long long>(tok0 + j) * p.ldo + (n >> 1)] = __float2bfloat16_rn(gate_f<EPI>(acc[j]) * other);
            }
        } else if (n < p.N) {
#pragma unroll
            for (int j = 0; j < MT; ++j) {
                if (j >= own) break;
                const long long idx = static_cast<long long>(tok0 + j) * p.ldo + n;
                if (EPI == VB200_EPI_ADD_F32 && j > 0 && j % kHeld == 0) load_held(j);
                if (EPI == VB200_EPI_RELU2) {
                    const float r = fmaxf(acc[j], 0.f);
                    static_cast<__nv_bfloat16*>(p.out)[idx] = __float2bfloat16_rn(r * r);
                } else if (EPI == VB200_EPI_BF16) static_cast<__nv_bfloat16*>(p.out)[idx] = __float2bfloat16_rn(acc[j]);
                else if (EPI == VB200_EPI_F32) static_cast<float*>(p.out)[idx] = acc[j];
                else {
                    const float hv = held[j % kHeld] + (p.addend != nullptr ? acc[j] + p.addend[idx] : acc[j]);
                    static_cast<float*>(p.out)[idx] = hv;
                    if (p.scaled_copy != nullptr)
                        static_cast<__nv_bfloat16*>(p.scaled_copy)[static_cast<long long>(tok0 + j) * p.N + n] = __float2bfloat16_rn(hv * gain);
                }
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) tmem_dealloc(tmem_base, C::kTmemCols);
    // a CTA exits with nothing on its way to it: it has counted all that the others send, except after an expired wait
    if (splits > 1 && *abort_flag) { __syncwarp(); cluster_arrive(); cluster_wait(); }
    abort_linger(abort_flag);
}

// ------------------------------------------------------------------------------------------------
// Host side
// ------------------------------------------------------------------------------------------------
using EncodeTiledFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn encode_fn() {
    static EncodeTiledFn fn = []() -> EncodeTiledFn {
        void* ptr = nullptr;
        cudaDriverEntryPointQueryResult qres;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &qres) != cudaSuccess) return nullptr;
        if (qres != cudaDriverEntryPointSuccess) return nullptr;
        return reinterpret_cast<EncodeTiledFn>(ptr);
    }();
    return fn;
}

// rows x K bf16 matrix with row stride ld (elements) -> 2-D map (K, rows), box [64][box_rows], 128-byte swizzle;
// reads past either extent return zeros.
int make_map_2d(CUtensorMap* m, const void* ptr, long long rows, long long K, long long ld, int box_rows) {
    EncodeTiledFn enc = encode_fn();
    if (!enc) return set_detail(VB200_ERR_CUDA, "cuTensorMapEncodeTiled is not available from the driver");
    cuuint64_t dims[2] = {static_cast<cuuint64_t>(K), static_cast<cuuint64_t>(rows)};
    cuuint64_t strides[1] = {static_cast<cuuint64_t>(ld) * 2};
    cuuint32_t box[2] = {static_cast<cuuint32_t>(kBK), static_cast<cuuint32_t>(box_rows)};
    cuuint32_t estr[2] = {1, 1};
    CUresult r = enc(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(ptr), dims, strides, box, estr,
                     CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                     CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) {
        static thread_local char buf[96];
        snprintf(buf, sizeof(buf), "cuTensorMapEncodeTiled (linear) failed with CUresult %d", static_cast<int>(r));
        return set_detail(VB200_ERR_CUDA, buf);
    }
    return VB200_OK;
}

// Raises the dynamic shared memory limit of one kernel instantiation once per device and thread;
// `configured` is the caller's (per instantiation) thread-local array of 64 markers, one per device ordinal.
template <typename Kernel>
int set_smem_once(Kernel kernel, int bytes, bool* configured) {
    int dev = 0;
    VB200_CUDA_TRY(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64) return set_detail(VB200_ERR_NO_DEVICE, "device ordinal out of range");
    if (!configured[dev]) {
        VB200_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes));
        configured[dev] = true;
    }
    return VB200_OK;
}

int sm_count(int* sms) {
    int dev = 0;
    VB200_CUDA_TRY(cudaGetDevice(&dev));
    VB200_CUDA_TRY(cudaDeviceGetAttribute(sms, cudaDevAttrMultiProcessorCount, dev));
    return VB200_OK;
}

template <int BN, int EPI, bool GROUPED = false>
int launch_wide(cudaStream_t s, const LinearParams& p) {
    using C = WideCfg<BN>;
    LinearMaps maps;
    if (int rc = make_map_2d(&maps.a, p.x, p.M, p.K, p.ldx, kTileA)) return rc;
    if (int rc = make_map_2d(&maps.b, p.w, GROUPED ? static_cast<long long>(p.groups) * p.group_rows : p.N, p.K, p.ldw, BN)) return rc;
    auto kernel = linear_wide_kernel<BN, EPI, GROUPED>;
    static thread_local bool configured[64] = {};
    if (int rc = set_smem_once(kernel, C::kSmemBytes, configured)) return rc;
    int sms = 0;
    if (int rc = sm_count(&sms)) return rc;
    const int tiles = (GROUPED ? p.group_tile_max : (p.M + kTileA - 1) / kTileA) * ((p.N + BN - 1) / BN);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(static_cast<unsigned>(tiles < sms ? tiles : sms));
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = C::kSmemBytes;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    VB200_CUDA_TRY(cudaLaunchKernelEx(&cfg, kernel, maps, p));
    note_launch();
    return VB200_OK;
}

template <int BN, int EPI>
int launch_pair(cudaStream_t s, const LinearParams& p, int sms) {
    using C = PairCfg<BN>;
    PairMaps maps;
    if (int rc = make_map_2d(&maps.a, p.x, p.M, p.K, p.ldx, kTileA)) return rc;
    if (int rc = make_map_2d(&maps.b, p.w, p.N, p.K, p.ldw, BN / 2)) return rc;
    auto kernel = linear_pair_kernel<BN, EPI>;
    static thread_local bool configured[64] = {};
    if (int rc = set_smem_once(kernel, C::kSmemBytes, configured)) return rc;
    const int tiles = ((p.M + 2 * kTileA - 1) / (2 * kTileA)) * ((p.N + BN - 1) / BN), pairs = sms / 2, last = tiles % pairs;
    // A last round that at most half of the pairs have a tile in is dealt out in halves of tiles; a half takes two thirds of a tile's time.  Whole tiles / halves,
    // weights from HBM: 3003 rows 2048 x 5632 60.2-62.1 / 53.3-58.4 us, 2048 x 2048 24-27 / 20.8-24.9, 11264 x 2048 94.4 / 91.6; 2100 rows 3072 x 2048
    // 24.2 / 21.9, 11264 x 2048 72.8 / 71.3; 1001 rows 11264 x 2048 36.8 / 35.7; 3500 rows 3072 x 2048 42.4-44.9 / 40.0-43.7, 11264 x 2048 107-116 / 105-114.
    const int whole = BN == 256 && tiles > pairs && 2 * last <= pairs ? tiles - last : tiles;
    maps.b_half = maps.b;                             // (the kernel reads it for halves only)
    if (whole < tiles)
        if (int rc = make_map_2d(&maps.b_half, p.w, p.N, p.K, p.ldw, BN / 4)) return rc;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(static_cast<unsigned>(2 * (tiles < pairs ? tiles : pairs)));
    cfg.blockDim = dim3(kPairThreads);
    cfg.dynamicSmemBytes = C::kSmemBytes;
    cfg.stream = s;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = 2;
    attr[1].val.clusterDim.y = 1;
    attr[1].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 2;
    VB200_CUDA_TRY(cudaLaunchKernelEx(&cfg, kernel, maps, p, whole));
    note_launch();
    return VB200_OK;
}

// More than 64 rows.  Pairs of CTAs with tiles of 256 columns; of 128 columns while one round over the SM pairs takes them all (768 rows, weights from
// HBM, 128 / 256 columns: 2048 x 2048 13.0 / 15.4 us, 2048 x 5632 23.5 / 31.8; with more rounds the wider tile is faster: 3003 rows, 11264 x 2048 118 / 92);
// single CTAs where the rows of a pair's last tile would be mostly padding and cost rounds (single / pairs: 300 rows, 11264 x 2048 17.9 / 22.7 us, 384 rows
// 18.1 / 22.8, though the pairs' last round is one of halves; 256 rows, which fill them, 18.2 / 17.0; 3003 rows 104.6 / 92.5).
template <int EPI>
int launch_many_rows(cudaStream_t s, const LinearParams& p) {
    int sms = 0;
    if (int rc = sm_count(&sms)) return rc;
    auto rounds = [&](int rows, int columns, int at_once) { return (((p.M + rows - 1) / rows) * ((p.N + columns - 1) / columns) + at_once - 1) / at_once; };
    if (rounds(2 * kTileA, 128, sms / 2) == 1) return launch_pair<128, EPI>(s, p, sms);
    const int pair = rounds(2 * kTileA, 256, sms / 2), single = rounds(kTileA, 256, sms);
    if (single * 4 < pair * 3) return launch_wide<256, EPI>(s, p);
    return launch_pair<256, EPI>(s, p, sms);
}

// K slices per tile of 128 rows: enough CTAs to touch every SM, equal slices when a nearby count allows it.  The slices fix the order in which a
// product's fp32 sums are added, so the count follows from N, K and the device alone and the same call keeps the same bits.  (Slices that minimise the K blocks
// of the busiest SM instead are faster at some sizes -- 8 tokens, 88 tiles x 32 blocks 3: 11.2 us against 2: 12.9 -- but sum in another order: the
// logits of whole models moved by 0.5 %, 2-8 % further from their 64-bit values.)
int pick_splits(int n_tiles, int k_blocks, int max_splits, int sms) {
    int want = (sms + n_tiles - 1) / n_tiles;
    if (want > max_splits) want = max_splits;
    if (want > k_blocks) want = k_blocks;
    if (want < 1) want = 1;
    for (int s = want; s <= max_splits && s <= k_blocks; ++s)
        if (k_blocks % s == 0) return s;
    return want;
}

template <int MT, int EPI>
int launch_skinny(cudaStream_t s, const LinearParams& p) {
    using C = SkinnyCfg<MT>;
    LinearMaps maps;
    if (int rc = make_map_2d(&maps.a, p.w, p.N, p.K, p.ldw, kTileA)) return rc;
    if (int rc = make_map_2d(&maps.b, p.x, p.M, p.K, p.ldx, MT)) return rc;
    auto kernel = linear_skinny_kernel<MT, EPI>;
    static thread_local bool configured[64] = {};
    if (int rc = set_smem_once(kernel, C::kSmemBytes, configured)) return rc;
    int sms = 0;
    if (int rc = sm_count(&sms)) return rc;
    const int n_tiles = (p.N + kTileA - 1) / kTileA;
    const int splits = p.splits > 0 ? (p.splits < C::kMaxSplits ? p.splits : C::kMaxSplits)
                                    : pick_splits(n_tiles, (p.K + kBK - 1) / kBK, C::kMaxSplits, sms);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(static_cast<unsigned>(n_tiles * splits));
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = C::kSmemBytes;
    cfg.stream = s;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    int n_attr = 1;
    if (splits > 1) {
        attr[1].id = cudaLaunchAttributeClusterDimension;
        attr[1].val.clusterDim.x = static_cast<unsigned>(splits);
        attr[1].val.clusterDim.y = 1;
        attr[1].val.clusterDim.z = 1;
        n_attr = 2;
    }
    cfg.attrs = attr;
    cfg.numAttrs = n_attr;
    VB200_CUDA_TRY(cudaLaunchKernelEx(&cfg, kernel, maps, p, splits));
    note_launch();
    return VB200_OK;
}

template <int EPI>
int launch_epi(cudaStream_t s, const LinearParams& p) {
    if (p.M <= 16) return launch_skinny<16, EPI>(s, p);
    if (p.M <= 32) return launch_skinny<32, EPI>(s, p);
    if (p.M <= 64) return launch_skinny<64, EPI>(s, p);
    return launch_many_rows<EPI>(s, p);
}

}  // namespace

int launch_linear_grouped(cudaStream_t s, const LinearParams& p) {
    switch (p.epilogue) {
        case VB200_EPI_BF16: return launch_wide<256, VB200_EPI_BF16, true>(s, p);
        case VB200_EPI_SWIGLU: return launch_wide<256, VB200_EPI_SWIGLU, true>(s, p);
        default: return set_detail(VB200_ERR_INVALID_ARG, "grouped linear: epilogue not available");
    }
}

int launch_linear(cudaStream_t s, const LinearParams& p) {
    switch (p.epilogue) {
        case VB200_EPI_BF16: return launch_epi<VB200_EPI_BF16>(s, p);
        case VB200_EPI_F32: return launch_epi<VB200_EPI_F32>(s, p);
        case VB200_EPI_ADD_F32: {
            if (int rc = launch_epi<VB200_EPI_ADD_F32>(s, p)) return rc;
            // the norm of the finished rows is a second launch, chained by programmatic dependent launch.  (Doing it
            // inside the weight-streaming kernel, by the CTA that finishes last, was measured: fence + ticket +
            // a lone CTA re-reading the rows cost 8 us on the decode step's critical path against 3-4 us here.)
            if (p.norm_out) return launch_rms_norm(s, static_cast<const float*>(p.out), p.norm_w, p.norm_out, p.M, p.N, p.norm_eps);
            return VB200_OK;
        }
        case VB200_EPI_SWIGLU: return launch_epi<VB200_EPI_SWIGLU>(s, p);
        case VB200_EPI_RELU2: return launch_epi<VB200_EPI_RELU2>(s, p);
        case VB200_EPI_REGLU: return launch_epi<VB200_EPI_REGLU>(s, p);
        default: return set_detail(VB200_ERR_INVALID_ARG, "unknown linear epilogue");
    }
}

}  // namespace vb200
