// Products of fp32 tiles in shared memory on the CUDA cores: the building blocks of the fp32 attention kernels
// (prefill_f32.cu, flash_bwd_f32.cu).
//
// Every product is issued as packed fma.rn.f32x2 (two IEEE fp32 FMAs per instruction).  A plain FMA per lane and cycle
// already fills an SM sub-partition's issue slot, which leaves none for the shared-memory loads; the packed form needs
// every other slot only.  128 threads compute one product as 8 (ty) x 16 (tx) threads:
//   tile_abt   C[64][64] += A[64][K] B[64][K]^T    thread: rows ty + 8 i, columns 4 tx + j; even and odd k in separate
//                                                  halves of an accumulator pair, so no operand has to be duplicated
//   tile_ab    C[64][N]  += A[64][64] B[64][N]     thread: rows ty + 8 i, columns 4 tx + 64 g; A values duplicated
//   (these two also with R = 4: 256 threads, rows ty + 16 i)
//   tile_atb   C[64][N]  += A[64][64]^T B[64][N]   thread: rows 8 ty + i, columns 4 tx + 64 g; A values duplicated
// An 8 x 4 (8 x 8) register block reads 12 (16) 16-byte words per 128 (256) FMAs: half (three eighths) of the
// shared-memory bandwidth at the full FMA rate; the 4 x 4 block that these kernels had before needed all of it.
//
// Tiles of B rows that tile_abt reads are swizzled: 16-byte word c of row r stands at word c ^ swz(r), so that the rows a
// quarter warp reads at one k fall into distinct banks without padding (which would not fit).
#pragma once

#include "common.cuh"

namespace vb200 {
namespace f32t {

constexpr int kTile = 64;              // rows of every tile
constexpr int kGroup = 128;            // threads that compute one product

using Pair = unsigned long long;       // two packed fp32 values

__device__ __forceinline__ void fma2(Pair& d, Pair a, Pair b) { asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(d) : "l"(a), "l"(b)); }
__device__ __forceinline__ void mul2(Pair& d, Pair a) { asm("mul.rn.f32x2 %0, %0, %1;" : "+l"(d) : "l"(a)); }
__device__ __forceinline__ Pair dup2(float x) {
    Pair r;
    asm("mov.b64 %0, {%1, %1};" : "=l"(r) : "f"(x));
    return r;
}
__device__ __forceinline__ float2 halves(Pair p) {
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(p));
    return r;
}
struct __align__(16) Quad { Pair lo, hi; };

// rows r of one 4-row block share the word swizzle of tile_abt's B operand (thread tx reads rows 4 tx + j); adjacent rows differ
// in the A operand's (rows ty and ty + 1 are read by one warp).  One function serves both: bits of r >> 2 and of r.
__device__ __forceinline__ int swz_b(int r) { return (r >> 2) & 7; }
__device__ __forceinline__ int swz_a(int r) { return r & 7; }

__device__ __forceinline__ void cp_async16(float* dst, const float* src, bool valid) {
    const int n = valid ? 16 : 0;      // 0: the 16 bytes become zeros, nothing is read
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(dst)), "l"(src), "r"(n) : "memory");
}
__device__ __forceinline__ void cp_async4(float* dst, const float* src, bool valid) {
    const int n = valid ? 4 : 0;
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(smem_u32(dst)), "l"(src), "r"(n) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_but_last() { asm volatile("cp.async.wait_group 1;" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

enum class Swizzle { None, A, B };

// 64 rows from row0 on (row stride ld elements, a multiple of 4; src 16-byte aligned) into a [64][DMAX] tile; rows from `rows`
// on become zeros, columns from D on stay as they are (no product reads them into a column that is kept).  All `threads` threads take part.
template <int DMAX, Swizzle SWZ>
__device__ __forceinline__ void load_rows(float* dst, const float* __restrict__ src, long long ld, int row0, int rows, int D, int tid, int threads) {
    constexpr int W = DMAX / 4;
    for (int i = tid; i < kTile * W; i += threads) {
        const int r = i / W, c = i % W;
        if (4 * c >= D) continue;
        const bool ok = row0 + r < rows;
        const int at = SWZ == Swizzle::None ? c : SWZ == Swizzle::A ? (c ^ swz_a(r)) : (c ^ swz_b(r));
        cp_async16(dst + r * DMAX + 4 * at, ok ? src + (row0 + r) * ld + 4 * c : src, ok);
    }
}

// s[i][j] = sum over words c < words of A[ty + 8 i] . B[4 tx + j]; A swizzled with swz_a, B with swz_b
template <int DMAX, int R = 8>
__device__ __forceinline__ void tile_abt(float (&s)[R][4], const float* A, const float* B, int words, int tx, int ty) {
    Pair acc[R][4];
#pragma unroll
    for (int i = 0; i < R; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = 0;
    const float* a0 = A + ty * DMAX;
    const float* b0 = B + 4 * tx * DMAX;
    const int sa = swz_a(ty), sb = swz_b(4 * tx);
#pragma unroll 2
    for (int c = 0; c < words; ++c) {
        const float* ap = a0 + 4 * (c ^ sa);
        const float* bp = b0 + 4 * (c ^ sb);
        Quad b[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) b[j] = *reinterpret_cast<const Quad*>(bp + j * DMAX);
#pragma unroll
        for (int i = 0; i < R; ++i) {
            const Quad a = *reinterpret_cast<const Quad*>(ap + kTile / R * i * DMAX);
#pragma unroll
            for (int j = 0; j < 4; ++j) fma2(acc[i][j], a.lo, b[j].lo);
#pragma unroll
            for (int j = 0; j < 4; ++j) fma2(acc[i][j], a.hi, b[j].hi);
        }
    }
#pragma unroll
    for (int i = 0; i < R; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const float2 h = halves(acc[i][j]);
            s[i][j] = h.x + h.y;
        }
}

// acc[i][2 g], acc[i][2 g + 1] (columns col0 + 4 tx + 64 g .. + 3) += sum over k0 <= kk < k1, in steps of 4, of A[ty + 8 i][kk] B[kk][...].
// A: row pitch PA; B: row pitch DMAX, swizzled with swz_b when SWZ.
template <int DMAX, int PA, int G, bool SWZ, int R = 8>
__device__ __forceinline__ void tile_ab(Pair (&acc)[R][2 * G], const float* A, const float* B, int k0, int k1, int col0, int tx, int ty) {
    const float* a0 = A + ty * PA;
#pragma unroll 2
    for (int kk = k0; kk < k1; kk += 4) {
        float4 a[R];
#pragma unroll
        for (int i = 0; i < R; ++i) a[i] = *reinterpret_cast<const float4*>(a0 + kTile / R * i * PA + kk);
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            Quad b[G];
#pragma unroll
            for (int g = 0; g < G; ++g) {
                const int word = (col0 >> 2) + tx + 16 * g;
                b[g] = *reinterpret_cast<const Quad*>(B + (kk + e) * DMAX + 4 * (SWZ ? (word ^ swz_b(kk)) : word));
            }
#pragma unroll
            for (int i = 0; i < R; ++i) {
                const Pair x = dup2(e == 0 ? a[i].x : e == 1 ? a[i].y : e == 2 ? a[i].z : a[i].w);
#pragma unroll
                for (int g = 0; g < G; ++g) { fma2(acc[i][2 * g], x, b[g].lo); fma2(acc[i][2 * g + 1], x, b[g].hi); }
            }
        }
    }
}

// acc[i][2 g], acc[i][2 g + 1] (columns 4 tx + 64 g .. + 3) += sum over r0 <= r < 64 of A[r][8 ty + i] B[r][...]; A: row pitch 64, B swizzled
// with swz_a
template <int DMAX, int G>
__device__ __forceinline__ void tile_atb(Pair (&acc)[8][2 * G], const float* A, const float* B, int tx, int ty, int r0 = 0) {
#pragma unroll 4
    for (int r = r0; r < kTile; ++r) {
        const float4 a0 = *reinterpret_cast<const float4*>(A + r * kTile + 8 * ty), a1 = *reinterpret_cast<const float4*>(A + r * kTile + 8 * ty + 4);
        const float a[8] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w};
        Quad b[G];
#pragma unroll
        for (int g = 0; g < G; ++g) b[g] = *reinterpret_cast<const Quad*>(B + r * DMAX + 4 * ((tx + 16 * g) ^ swz_a(r)));
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const Pair x = dup2(a[i]);
#pragma unroll
            for (int g = 0; g < G; ++g) { fma2(acc[i][2 * g], x, b[g].lo); fma2(acc[i][2 * g + 1], x, b[g].hi); }
        }
    }
}

// The two products above for the tile on the diagonal of a causal mask, where A[r][c] with c > r stands for a position that is not seen: those are
// left out, not multiplied by zero -- a row of B that holds an infinity would reach every row of the tile as 0 * inf.
template <int DMAX, int PA, int K0, int KN>
__device__ __forceinline__ void tile_ab_lower(Pair (&acc)[8][2], const float* A, const float* B, int col0, int tx, int ty) {
    const float* a0 = A + ty * PA;
#pragma unroll
    for (int kk = K0; kk < K0 + KN; kk += 4) {
        const int q = kk >> 3;                            // row ty + 8 q sees kk + e up to its own place; the rows of later i see all of this octet
        float4 a[8];
#pragma unroll
        for (int i = q; i < 8; ++i) a[i] = *reinterpret_cast<const float4*>(a0 + 8 * i * PA + kk);
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const Quad b = *reinterpret_cast<const Quad*>(B + (kk + e) * DMAX + 4 * (((col0 >> 2) + tx) ^ swz_b(kk)));
#pragma unroll
            for (int i = q; i < 8; ++i) {
                if (i == q && (kk & 7) + e > ty) continue;
                const Pair x = dup2(e == 0 ? a[i].x : e == 1 ? a[i].y : e == 2 ? a[i].z : a[i].w);
                fma2(acc[i][0], x, b.lo);
                fma2(acc[i][1], x, b.hi);
            }
        }
    }
}

template <int DMAX, int G>
__device__ __forceinline__ void tile_atb_lower(Pair (&acc)[8][2 * G], const float* A, const float* B, int tx, int ty) {
#pragma unroll
    for (int m = 0; m < 8; ++m) {                         // rows 8 ty + m see columns 8 ty .. 8 ty + m
        const int r = 8 * ty + m;
        const float4 a0 = *reinterpret_cast<const float4*>(A + r * kTile + 8 * ty), a1 = *reinterpret_cast<const float4*>(A + r * kTile + 8 * ty + 4);
        const float a[8] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w};
#pragma unroll
        for (int g = 0; g < G; ++g) {
            const Quad b = *reinterpret_cast<const Quad*>(B + r * DMAX + 4 * ((tx + 16 * g) ^ swz_a(r)));
#pragma unroll
            for (int i = 0; i <= m; ++i) {
                const Pair x = dup2(a[i]);
                fma2(acc[i][2 * g], x, b.lo);
                fma2(acc[i][2 * g + 1], x, b.hi);
            }
        }
    }
    tile_atb<DMAX, G>(acc, A, B, tx, ty, 8 * ty + 8);
}

__device__ __forceinline__ float4 quad4(Pair lo, Pair hi) {
    const float2 a = halves(lo), b = halves(hi);
    return make_float4(a.x, a.y, b.x, b.y);
}

}  // namespace f32t
}  // namespace vb200
