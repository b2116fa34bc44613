// Flash-attention backward in fp32 (the dtype of the reference's training path): dQ, dK, dV from the
// saved output and log-sum-exp, recomputing P tile by tile -- flash_attention_backward_cpu_dispatch,
// src/ops/flash_attention.cpp:366-482, without dropout:
//   Di = rowsum(dO * O);  P = exp(scale Q K^T - LSE);  dV = P^T dO;  dS = P * (dO V^T - Di);
//   dQ = scale dS K;  dK = scale dS^T Q.
// Three launches, all deterministic (no atomics): the row sums; one CTA per 64-key tile walking the query
// tiles that see it (dK, dV in registers); one CTA per 64-query tile walking its key tiles (dQ in registers).
// Head dims of 64 and 128 above 64 positions run on the tensor cores instead (attention_f32_sm100.cu), given the workspace.
// CUDA cores, 64 x 64 tiles, products as in f32_tiles.cuh.  A CTA is two groups of 128 threads that hold the same
// positions of a tile: one computes S and P, the other dO V^T and dS, at the same time; then one accumulates dV while the
// other accumulates dK (or each one half of dQ's columns).  That keeps the register blocks at 8 x 4 and 8 x 8 -- with all
// 256 threads on one product after the other they would be half as large, and shared memory the bound.  The streamed
// tiles are double-buffered, which with head_dim 128 takes all of an SM's shared memory: one CTA per SM.
#include "f32_tiles.cuh"
#include "kernels.h"
#include "hybrid.cuh"

namespace vb200 {
namespace {

using namespace f32t;

constexpr int kT = 32;                 // tile edge of the general kernels
constexpr int kBwdThreads = 256;
constexpr int kPitchDs = kTile + 4;    // dS in the dQ kernel: rows ty and ty + 1 of one warp in distinct banks

// barrier of the 128 threads of one group
template <int GROUP> __device__ __forceinline__ void group_sync() { asm volatile("bar.sync %0, %1;" ::"n"(GROUP + 1), "n"(kGroup) : "memory"); }

__global__ void bwd_delta_kernel(const float* __restrict__ d_out, const float* __restrict__ out, float* __restrict__ delta,
                                 long long rows, int D) {
    const long long row = blockIdx.x * static_cast<long long>(blockDim.x / 32) + (threadIdx.x >> 5);
    if (row >= rows) return;
    const int lane = threadIdx.x & 31;
    float s = 0.f;
    for (int d = lane; d < D; d += 32) s += d_out[row * D + d] * out[row * D + d];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xFFFFFFFFu, s, o);
    if (lane == 0) delta[row] = s;
}

// dynamic shared memory, in floats: two resident tiles, two double-buffered ones, their rows' LSE and Di, P and dS
template <int DMAX> constexpr int dkdv_floats() { return 6 * kTile * DMAX + 2 * kTile * kTile + 4 * kTile; }
template <int DMAX> constexpr int dq_floats() { return 6 * kTile * DMAX + kTile * kPitchDs + 2 * kTile; }

// p = exp(s scale - LSE) of the visible positions of one thread's 8 x 4 block (queries i0 + ty + 8 i, keys j0 + 4 tx + j)
__device__ __forceinline__ void weights(float (&s)[8][4], const float* Ls, int i0, int j0, int N, float scale, int causal, int tx, int ty) {
    const bool edge = i0 + kTile > N || j0 + kTile > N || (causal && j0 + kTile - 1 > i0);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int gi = i0 + ty + 8 * i;
        const float l = Ls[ty + 8 * i];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const float w = expf(s[i][j] * scale - l);
            const int gj = j0 + 4 * tx + j;
            s[i][j] = !edge || (gi < N && gj < N && (!causal || gj <= gi)) ? w : 0.f;
        }
    }
}

template <int DMAX>
__global__ void __launch_bounds__(kBwdThreads, 1)
bwd_dkdv_kernel(AttnBwdParams p) {
    extern __shared__ __align__(16) float sm[];
    constexpr int G = DMAX / 64, kRows = kTile * DMAX;
    float* Ks = sm; float* Vs = Ks + kRows;
    float* Qs = Vs + kRows;                       // [2]
    float* dOs = Qs + 2 * kRows;                  // [2]
    float* Ps = dOs + 2 * kRows; float* dSs = Ps + kTile * kTile;
    float* Ls = dSs + kTile * kTile;              // [2][64]
    float* Dis = Ls + 2 * kTile;                  // [2][64]
    const int D = p.D, N = p.N, words = D >> 2;
    const int group = threadIdx.x / kGroup, t = threadIdx.x % kGroup, tx = t & 15, ty = t >> 4;
    const int j0 = blockIdx.y * kTile;            // the key tiles with the most query tiles are launched first
    const long long bh = blockIdx.x;
    const float* q = p.q + bh * N * D; const float* k = p.k + bh * N * D; const float* v = p.v + bh * N * D;
    const float* d_out = p.d_out + bh * N * D; const float* lse = p.lse + bh * N; const float* delta = p.delta + bh * N;

    auto load_queries = [&](int i0, int buf) {
        load_rows<DMAX, Swizzle::A>(group == 0 ? Qs + buf * kRows : dOs + buf * kRows, group == 0 ? q : d_out, D, i0, N, D, t, kGroup);
        if (t < kTile) {
            const bool ok = i0 + t < N;
            const float* src = group == 0 ? lse : delta;
            cp_async4((group == 0 ? Ls : Dis) + buf * kTile + t, ok ? src + i0 + t : src, ok);
        }
        cp_async_commit();
    };
    load_rows<DMAX, Swizzle::B>(group == 0 ? Ks : Vs, group == 0 ? k : v, D, j0, N, D, t, kGroup);
    const int i_first = p.causal ? j0 : 0;        // query tiles before the key tile see none of it
    load_queries(i_first, 0);

    Pair acc[8][2 * G];                           // group 0: dV, group 1: dK; keys 8 ty + i
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int g = 0; g < 2 * G; ++g) acc[i][g] = 0;

    int buf = 0;
    for (int i0 = i_first; i0 < N; i0 += kTile, buf ^= 1) {
        cp_async_wait_all();
        __syncthreads();                          // this query tile has arrived; the previous one, its P and dS are consumed
        if (i0 + kTile < N) load_queries(i0 + kTile, buf ^ 1);
        float s[8][4];
        tile_abt<DMAX>(s, (group == 0 ? Qs : dOs) + buf * kRows, group == 0 ? Ks : Vs, words, tx, ty);
        if (group == 0) {
            weights(s, Ls + buf * kTile, i0, j0, N, p.scale, p.causal, tx, ty);
#pragma unroll
            for (int i = 0; i < 8; ++i) *reinterpret_cast<float4*>(Ps + (ty + 8 * i) * kTile + 4 * tx) = make_float4(s[i][0], s[i][1], s[i][2], s[i][3]);
        }
        __syncthreads();                          // P is complete
        if (group == 1) {
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const float4 w = *reinterpret_cast<const float4*>(Ps + (ty + 8 * i) * kTile + 4 * tx);
                const float di = Dis[buf * kTile + ty + 8 * i];
                *reinterpret_cast<float4*>(dSs + (ty + 8 * i) * kTile + 4 * tx) =
                    make_float4(w.x * (s[i][0] - di), w.y * (s[i][1] - di), w.z * (s[i][2] - di), w.w * (s[i][3] - di));
            }
            group_sync<1>();
        }
        const float* weights_of = group == 0 ? Ps : dSs;
        const float* rows_of = (group == 0 ? dOs : Qs) + buf * kRows;
        if (p.causal && i0 == j0) tile_atb_lower<DMAX, G>(acc, weights_of, rows_of, tx, ty);
        else tile_atb<DMAX, G>(acc, weights_of, rows_of, tx, ty);
    }
    float* out = group == 0 ? p.dv : p.dk;
    const float scale = group == 0 ? 1.f : p.scale;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int gj = j0 + 8 * ty + i;
        if (gj >= N) continue;
#pragma unroll
        for (int g = 0; g < G; ++g) {
            const int d = 4 * tx + 64 * g;
            if (d < D) {
                const float4 x = quad4(acc[i][2 * g], acc[i][2 * g + 1]);
                *reinterpret_cast<float4*>(out + (bh * N + gj) * D + d) = make_float4(x.x * scale, x.y * scale, x.z * scale, x.w * scale);
            }
        }
    }
}

// dQ of a half of the columns per group: with DMAX 64 both groups would hold 32 columns, too few for a 4-column block per
// thread, so there each group takes half of the keys of a tile instead, and the halves are added at the end.
template <int DMAX>
__global__ void __launch_bounds__(kBwdThreads, 1)
bwd_dq_kernel(AttnBwdParams p) {
    extern __shared__ __align__(16) float sm[];
    constexpr int kRows = kTile * DMAX;
    float* Qs = sm; float* dOs = Qs + kRows;
    float* Ks = dOs + kRows;                      // [2]
    float* Vs = Ks + 2 * kRows;                   // [2]
    float* dSs = Vs + 2 * kRows;                  // P, then dS
    float* Ls = dSs + kTile * kPitchDs; float* Dis = Ls + kTile;
    const int D = p.D, N = p.N, words = D >> 2;
    const int group = threadIdx.x / kGroup, t = threadIdx.x % kGroup, tx = t & 15, ty = t >> 4;
    const int i0 = (gridDim.y - 1 - blockIdx.y) * kTile;      // causal: the query tiles with the most key tiles first
    const long long bh = blockIdx.x;
    const float* q = p.q + bh * N * D; const float* k = p.k + bh * N * D; const float* v = p.v + bh * N * D;
    const float* d_out = p.d_out + bh * N * D; const float* lse = p.lse + bh * N; const float* delta = p.delta + bh * N;

    auto load_keys = [&](int j0, int buf) {
        load_rows<DMAX, Swizzle::B>(group == 0 ? Ks + buf * kRows : Vs + buf * kRows, group == 0 ? k : v, D, j0, N, D, t, kGroup);
        cp_async_commit();
    };
    load_rows<DMAX, Swizzle::A>(group == 0 ? Qs : dOs, group == 0 ? q : d_out, D, i0, N, D, t, kGroup);
    if (t < kTile) {
        const bool ok = i0 + t < N;
        const float* src = group == 0 ? lse : delta;
        cp_async4((group == 0 ? Ls : Dis) + t, ok ? src + i0 + t : src, ok);
    }
    load_keys(0, 0);

    Pair acc[8][2];                               // queries ty + 8 i
#pragma unroll
    for (int i = 0; i < 8; ++i) acc[i][0] = acc[i][1] = 0;

    const int j_end = p.causal ? min(N, i0 + kTile) : N;      // key tiles past the query tile are invisible
    int buf = 0;
    for (int j0 = 0; j0 < j_end; j0 += kTile, buf ^= 1) {
        cp_async_wait_all();
        __syncthreads();                          // this key tile has arrived; the previous one and its dS are consumed
        if (j0 + kTile < j_end) load_keys(j0 + kTile, buf ^ 1);
        float s[8][4];
        tile_abt<DMAX>(s, group == 0 ? Qs : dOs, (group == 0 ? Ks : Vs) + buf * kRows, words, tx, ty);
        if (group == 0) {
            weights(s, Ls, i0, j0, N, p.scale, p.causal, tx, ty);
#pragma unroll
            for (int i = 0; i < 8; ++i) *reinterpret_cast<float4*>(dSs + (ty + 8 * i) * kPitchDs + 4 * tx) = make_float4(s[i][0], s[i][1], s[i][2], s[i][3]);
        }
        __syncthreads();                          // P is complete
        if (group == 1) {
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                float4* at = reinterpret_cast<float4*>(dSs + (ty + 8 * i) * kPitchDs + 4 * tx);
                const float4 w = *at;
                const float di = Dis[ty + 8 * i];
                *at = make_float4(w.x * (s[i][0] - di), w.y * (s[i][1] - di), w.z * (s[i][2] - di), w.w * (s[i][3] - di));
            }
        }
        __syncthreads();                          // dS is complete
        if (p.causal && j0 == i0) {
            if (DMAX == 128) tile_ab_lower<DMAX, kPitchDs, 0, kTile>(acc, dSs, Ks + buf * kRows, 64 * group, tx, ty);
            else if (group == 0) tile_ab_lower<DMAX, kPitchDs, 0, kTile / 2>(acc, dSs, Ks + buf * kRows, 0, tx, ty);
            else tile_ab_lower<DMAX, kPitchDs, kTile / 2, kTile / 2>(acc, dSs, Ks + buf * kRows, 0, tx, ty);
        } else if (DMAX == 128) tile_ab<DMAX, kPitchDs, 1, true>(acc, dSs, Ks + buf * kRows, 0, kTile, 64 * group, tx, ty);
        else tile_ab<DMAX, kPitchDs, 1, true>(acc, dSs, Ks + buf * kRows, group * (kTile / 2), (group + 1) * (kTile / 2), 0, tx, ty);
    }
    if (DMAX == 64) {
        __syncthreads();                          // every tile is consumed: the second half of the keys passes its sums through Qs
        float4* half = reinterpret_cast<float4*>(Qs);
        if (group == 1) {
#pragma unroll
            for (int i = 0; i < 8; ++i) half[i * kGroup + t] = quad4(acc[i][0], acc[i][1]);
        }
        __syncthreads();
        if (group == 1) return;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const float4 x = quad4(acc[i][0], acc[i][1]), y = half[i * kGroup + t];
            const int gi = i0 + ty + 8 * i, d = 4 * tx;
            if (gi < N && d < D)
                *reinterpret_cast<float4*>(p.dq + (bh * N + gi) * D + d) =
                    make_float4((x.x + y.x) * p.scale, (x.y + y.y) * p.scale, (x.z + y.z) * p.scale, (x.w + y.w) * p.scale);
        }
        return;
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int gi = i0 + ty + 8 * i, d = 4 * tx + 64 * group;
        if (gi < N && d < D) {
            const float4 x = quad4(acc[i][0], acc[i][1]);
            *reinterpret_cast<float4*>(p.dq + (bh * N + gi) * D + d) = make_float4(x.x * p.scale, x.y * p.scale, x.z * p.scale, x.w * p.scale);
        }
    }
}

// ---- any head_dim up to 128 and 4-byte alignment: 32 x 32 tiles, scalar loads, rows padded by one float ----

// rows [r0, r0 + 32) of a [N, D] matrix into a padded tile; rows past N become zeros
__device__ __forceinline__ void load_tile(float* dst, const float* __restrict__ src, int r0, int N, int D, int ld) {
    for (int idx = threadIdx.x; idx < kT * D; idx += kBwdThreads) {
        const int r = idx / D, d = idx - r * D;
        dst[r * ld + d] = (r0 + r < N) ? src[static_cast<long long>(r0 + r) * D + d] : 0.f;
    }
}

// p and ds of the (query tile i0, key tile j0) pair: thread t owns query i0 + t/8 and keys j0 + 4 (t%8) .. + 3
__device__ __forceinline__ void tile_p_ds(const float* Qs, const float* Ks, const float* Vs, const float* dOs, const float* Ls,
                                          const float* Dis, float* Ps, float* dSs, int i0, int j0, int N, int D, int ld,
                                          float scale, int causal) {
    const int i = threadIdx.x >> 3, jb = (threadIdx.x & 7) * 4;
    float s[4] = {0.f, 0.f, 0.f, 0.f}, dp[4] = {0.f, 0.f, 0.f, 0.f};
    for (int d = 0; d < D; ++d) {
        const float qv = Qs[i * ld + d], gv = dOs[i * ld + d];
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            s[c] = fmaf(qv, Ks[(jb + c) * ld + d], s[c]);
            dp[c] = fmaf(gv, Vs[(jb + c) * ld + d], dp[c]);
        }
    }
#pragma unroll
    for (int c = 0; c < 4; ++c) {
        const int gi = i0 + i, gj = j0 + jb + c;
        const bool visible = gi < N && gj < N && (!causal || gj <= gi);
        const float p = visible ? expf(s[c] * scale - Ls[i]) : 0.f;
        Ps[i * (kT + 1) + jb + c] = p;
        dSs[i * (kT + 1) + jb + c] = p * (dp[c] - Dis[i]);
    }
}

template <int DMAX>
__global__ void __launch_bounds__(kBwdThreads)
bwd_dkdv_any_kernel(AttnBwdParams p) {
    extern __shared__ float sm[];
    const int D = p.D, ld = D + 1, N = p.N;
    float* Ks = sm; float* Vs = Ks + kT * ld; float* Qs = Vs + kT * ld; float* dOs = Qs + kT * ld;
    float* Ps = dOs + kT * ld; float* dSs = Ps + kT * (kT + 1); float* Ls = dSs + kT * (kT + 1); float* Dis = Ls + kT;
    const int j0 = blockIdx.x * kT;
    const long long bh = static_cast<long long>(blockIdx.z) * p.H + blockIdx.y;
    const float* q = p.q + bh * N * D; const float* k = p.k + bh * N * D; const float* v = p.v + bh * N * D;
    const float* d_out = p.d_out + bh * N * D; const float* lse = p.lse + bh * N; const float* delta = p.delta + bh * N;
    load_tile(Ks, k, j0, N, D, ld);
    load_tile(Vs, v, j0, N, D, ld);
    // thread t accumulates key j0 + t/8, dims (t%8) + 8 m
    const int j = threadIdx.x >> 3, dl = threadIdx.x & 7;
    float dk[DMAX / 8], dv[DMAX / 8];
#pragma unroll
    for (int m = 0; m < DMAX / 8; ++m) { dk[m] = 0.f; dv[m] = 0.f; }
    const int i_first = p.causal ? j0 : 0;                      // query tiles before the key tile see none of it
    for (int i0 = i_first; i0 < N; i0 += kT) {
        __syncthreads();
        load_tile(Qs, q, i0, N, D, ld);
        load_tile(dOs, d_out, i0, N, D, ld);
        if (threadIdx.x < kT) {
            const int gi = i0 + threadIdx.x;
            Ls[threadIdx.x] = gi < N ? lse[gi] : 0.f;
            Dis[threadIdx.x] = gi < N ? delta[gi] : 0.f;
        }
        __syncthreads();
        tile_p_ds(Qs, Ks, Vs, dOs, Ls, Dis, Ps, dSs, i0, j0, N, D, ld, p.scale, p.causal);
        __syncthreads();
        for (int i = 0; i < kT; ++i) {
            const float pv = Ps[i * (kT + 1) + j], ds = dSs[i * (kT + 1) + j];
#pragma unroll
            for (int m = 0; m < DMAX / 8; ++m) {
                const int d = dl + 8 * m;
                if (d < D) {
                    dv[m] = fmaf(pv, dOs[i * ld + d], dv[m]);
                    dk[m] = fmaf(ds, Qs[i * ld + d], dk[m]);
                }
            }
        }
    }
    if (j0 + j < N) {
#pragma unroll
        for (int m = 0; m < DMAX / 8; ++m) {
            const int d = dl + 8 * m;
            if (d < D) {
                p.dk[(bh * N + j0 + j) * D + d] = dk[m] * p.scale;
                p.dv[(bh * N + j0 + j) * D + d] = dv[m];
            }
        }
    }
}

template <int DMAX>
__global__ void __launch_bounds__(kBwdThreads)
bwd_dq_any_kernel(AttnBwdParams p) {
    extern __shared__ float sm[];
    const int D = p.D, ld = D + 1, N = p.N;
    float* Ks = sm; float* Vs = Ks + kT * ld; float* Qs = Vs + kT * ld; float* dOs = Qs + kT * ld;
    float* Ps = dOs + kT * ld; float* dSs = Ps + kT * (kT + 1); float* Ls = dSs + kT * (kT + 1); float* Dis = Ls + kT;
    const int i0 = blockIdx.x * kT;
    const long long bh = static_cast<long long>(blockIdx.z) * p.H + blockIdx.y;
    const float* q = p.q + bh * N * D; const float* k = p.k + bh * N * D; const float* v = p.v + bh * N * D;
    const float* d_out = p.d_out + bh * N * D; const float* lse = p.lse + bh * N; const float* delta = p.delta + bh * N;
    load_tile(Qs, q, i0, N, D, ld);
    load_tile(dOs, d_out, i0, N, D, ld);
    if (threadIdx.x < kT) {
        const int gi = i0 + threadIdx.x;
        Ls[threadIdx.x] = gi < N ? lse[gi] : 0.f;
        Dis[threadIdx.x] = gi < N ? delta[gi] : 0.f;
    }
    const int i = threadIdx.x >> 3, dl = threadIdx.x & 7;
    float dq[DMAX / 8];
#pragma unroll
    for (int m = 0; m < DMAX / 8; ++m) dq[m] = 0.f;
    const int j_end = p.causal ? min(N, i0 + kT) : N;           // key tiles past the query tile are invisible
    for (int j0 = 0; j0 < j_end; j0 += kT) {
        __syncthreads();
        load_tile(Ks, k, j0, N, D, ld);
        load_tile(Vs, v, j0, N, D, ld);
        __syncthreads();
        tile_p_ds(Qs, Ks, Vs, dOs, Ls, Dis, Ps, dSs, i0, j0, N, D, ld, p.scale, p.causal);
        __syncthreads();
        for (int jj = 0; jj < kT; ++jj) {
            const float ds = dSs[i * (kT + 1) + jj];
#pragma unroll
            for (int m = 0; m < DMAX / 8; ++m) {
                const int d = dl + 8 * m;
                if (d < D) dq[m] = fmaf(ds, Ks[jj * ld + d], dq[m]);
            }
        }
    }
    if (i0 + i < N) {
#pragma unroll
        for (int m = 0; m < DMAX / 8; ++m) {
            const int d = dl + 8 * m;
            if (d < D) p.dq[(bh * N + i0 + i) * D + d] = dq[m] * p.scale;
        }
    }
}

size_t any_smem_bytes(int D) { return sizeof(float) * (4 * kT * (D + 1) + 2 * kT * (kT + 1) + 2 * kT); }

// The attribute belongs to the device's context: raised once per device ordinal, thread and kernel.
template <typename Kernel>
int set_smem_once(Kernel kernel, size_t bytes, bool* configured) {
    int dev = 0;
    VB200_CUDA_TRY(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64) return set_detail(VB200_ERR_NO_DEVICE, "device ordinal out of range");
    if (!configured[dev]) {
        VB200_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(bytes)));
        configured[dev] = true;
    }
    return VB200_OK;
}

template <int DMAX>
int launch_bwd_any(cudaStream_t s, const AttnBwdParams& p) {
    static thread_local bool c1[64] = {}, c2[64] = {};
    if (int rc = set_smem_once(bwd_dkdv_any_kernel<DMAX>, any_smem_bytes(DMAX), c1)) return rc;
    if (int rc = set_smem_once(bwd_dq_any_kernel<DMAX>, any_smem_bytes(DMAX), c2)) return rc;
    dim3 grid(static_cast<unsigned>((p.N + kT - 1) / kT), static_cast<unsigned>(p.H), static_cast<unsigned>(p.B));
    bwd_dkdv_any_kernel<DMAX><<<grid, kBwdThreads, any_smem_bytes(p.D), s>>>(p);
    bwd_dq_any_kernel<DMAX><<<grid, kBwdThreads, any_smem_bytes(p.D), s>>>(p);
    return VB200_OK;
}

template <int DMAX>
int launch_bwd_tiled(cudaStream_t s, const AttnBwdParams& p) {
    constexpr size_t m1 = sizeof(float) * dkdv_floats<DMAX>(), m2 = sizeof(float) * dq_floats<DMAX>();
    static thread_local bool c1[64] = {}, c2[64] = {};
    if (int rc = set_smem_once(bwd_dkdv_kernel<DMAX>, m1, c1)) return rc;
    if (int rc = set_smem_once(bwd_dq_kernel<DMAX>, m2, c2)) return rc;
    dim3 grid(static_cast<unsigned>(p.B) * static_cast<unsigned>(p.H), static_cast<unsigned>((p.N + kTile - 1) / kTile));
    bwd_dkdv_kernel<DMAX><<<grid, kBwdThreads, m1, s>>>(p);
    bwd_dq_kernel<DMAX><<<grid, kBwdThreads, m2, s>>>(p);
    return VB200_OK;
}

// 16-byte rows: the tiled kernels, except where most of a 64 x 64 tile would be padding and the general kernels' 32 x 32 tiles, several CTAs of which
// share an SM, finish first (general / tiled, causal): up to 32 positions with head_dim up to 32 (one head, 32 x 32: 16.9 / 18.9 us), or with more heads than
// SMs (256 heads, 32 x 64: 34.6 / 44.6 us; 1024 heads, 16 x 128: 202 / 226, but 32 x 128: 241 / 232); 65 to 96 positions of many narrow heads (1024 heads,
// 65 x 8: 233 / 272 us, 65 x 16: 271 / 289, 65 x 32: 343 / 325; not causal 64 x 8 of 200 heads 83 / 76).  (A grid's second dimension ends at 65535, far above
// any sequence that fits the device.)
bool rows_aligned(const AttnBwdParams& p) {
    auto aligned = [](const void* x) { return reinterpret_cast<uintptr_t>(x) % 16 == 0; };
    return p.D % 4 == 0 && aligned(p.d_out) && aligned(p.q) && aligned(p.k) && aligned(p.v) && aligned(p.dq) && aligned(p.dk) && aligned(p.dv);
}
bool tiled_ok(const AttnBwdParams& p) {
    if (!rows_aligned(p) || (p.N + kTile - 1) / kTile > 65535) return false;
    const long long heads = static_cast<long long>(p.B) * p.H, sms = device_sm_count();
    if (p.N <= kT) return p.D > 32 && (heads <= sms || p.D > (p.N <= 16 ? 128 : 64));
    return !(p.causal && p.N > kTile && p.N <= 3 * kT && p.D <= 16 && heads > 2 * sms);
}

}  // namespace

// The tensor cores (attention_f32_sm100.cu) from the second block of 64 positions on.  These kernels / those: 16 heads, 512 x 64 127 / 36 us; 16, 2048 x 128
// 1595 / 439; 1024, 96 x 64 416 / 246; one head, 65 x 64 45 / 14; but 1024 heads, 64 x 64 167 / 187, 256 heads, 64 x 128 91 / 100.
bool attention_bwd_f32_on_tensor_cores(int D, int N) {
    return (D == 64 || D == 128) && N > 64;
}

int launch_attention_bwd_f32(cudaStream_t s, const AttnBwdParams& p) {
    if (p.D > 128) return set_detail(VB200_ERR_UNSUPPORTED, "attention backward supports head_dim <= 128");
    if (p.split != nullptr && rows_aligned(p) && reinterpret_cast<uintptr_t>(p.out) % 16 == 0) return launch_attention_bwd_f32_sm100(s, p, p.split);
    const long long rows = static_cast<long long>(p.B) * p.H * p.N;
    bwd_delta_kernel<<<static_cast<unsigned>((rows + 7) / 8), 256, 0, s>>>(p.d_out, p.out, p.delta, rows, p.D);
    const int rc = tiled_ok(p) ? (p.D <= 64 ? launch_bwd_tiled<64>(s, p) : launch_bwd_tiled<128>(s, p))
                               : (p.D <= 64 ? launch_bwd_any<64>(s, p) : launch_bwd_any<128>(s, p));
    if (rc != VB200_OK) return rc;
    note_launch(3);
    VB200_CUDA_TRY(cudaPeekAtLastError());
    return VB200_OK;
}

}  // namespace vb200
