// fp32 attention, forward and backward, on the tensor cores without giving up fp32: every fp32 operand is the exact sum of three
// bf16 terms (8 significant bits each), and a product of two operands is the six bf16 products whose terms are at least 2^-18 of
// it.  What is left out is 2^-26 of a product, below the rounding of an fp32 FMA.
//
// One kernel body, four uses.  A CTA owns 128 rows of one (batch, head) and walks the other sequence side in blocks of 64 rows:
//
//             rows A1, A2   blocks B1, B2     X = A1 B1^T      Y = A2 B2^T      W                                   sum
//   forward   Q             K, V              scores           -                exp(X - running max)                W B2
//   dV        K             Q, dO             scores^T         -                exp(X scale - LSE)                  W B2
//   dQ        Q, dO         K, V              scores           dO V^T           exp(X scale - LSE) (Y - Di)         W B1
//   dK        K, V          Q, dO             scores^T         V dO^T           exp(X scale - LSE) (Y - Di)         W B1
//
//   warps 0-3    W of one block, a row per thread; split into its three terms in tensor memory
//   warps 4-7    the sum, a row per thread, in registers
//   warp  8      bulk copies of blocks into a shared-memory ring
//   warp  9      tcgen05.mma issuer, TMEM owner
//
// The terms of the streamed operands are written to the workspace beforehand (split_blocks_kernel), each block as it will stand in
// shared memory: splitting them where they are used repeats the work for every tile of rows that reads them, and eight warps that did
// so were what the kernel waited for (2 x 16 x 1999 x 128: forward 278 us, backward 1086; calls now 197 and 860-950, splits included).
//
// What bounds it: with head_dim 128 the products, 48 of 64 columns and 24 of 128 per block in the forward, beside the weights of one warpgroup (tensor
// pipe busy 64 % of the forward's time, 57 % of the backward's, 16 x 2048 x 128); in dQ and dK also the wait for W, whose slot TMEM holds only once.
// The same calls on the CUDA cores (prefill_f32.cu, flash_bwd_f32.cu): 1105 and 3087 us; 16 x 512 x 64 50 and 128 us against 21 and 36-40.
//
// The tensor cores add with truncation, so no sum stays with them for long: a block's six products are added smallest first, and
// each block's result is added to the sum in registers, rounded to nearest.  What the last eight (or four) additions of a score lose
// on average is given back by factors (Loss).  A1 (and of A2 what fits) is read from TMEM: an
// operand of 64 columns from shared memory would make the product wait for the 128 rows of A.
//
// TMEM columns: A1 [3 D/2], A2 [terms in TMEM], per slot X [64] (and Y [64]) overwritten by the terms of W [96], the block sum [D].
//
// Numbers outside 2^-100 .. 2^126 (or inf, NaN; zeros are fine) have terms that bf16 does not hold, and 0 * inf of a masked position would
// reach every row of a tile: a CTA that meets one element of that kind in its rows or blocks computes its rows again on the CUDA cores
// (plain_rows), in the order of a plain loop.  Weights are not looked at: below 2^-100 they lose bits that matter only to a row without larger ones.
#include "kernels.h"
#include "hybrid.cuh"

namespace vb200 {
namespace {

constexpr int kRows = 128, kCols = 64;
constexpr int kLoadWarp = 8, kIssueWarp = 9;
constexpr int kThreads = (kIssueWarp + 1) * 32;
constexpr float kLn2 = 0.6931471805599453f;
constexpr float kLeast = 0x1p-100f;
// What the truncating additions lose on average, given back by factors of the scores (X), of dO V^T and V dO^T (Y), and of the results.  Fitted to the
// slopes of O, LSE, dQ, dK and dV against 64 bits over 64 to 2048 normal rows, -3e-7 .. -3e-8 without them and within 4e-8 with them; Y's also to rows with
// a common offset, whose Y - Di cancels.  X's stands in the second factor of the exponent (forward) and in the exponent itself (backward), not in
// the scale, where it would be a whole step of a float and the backward's X another one than the forward's.  Error against that of the
// CUDA cores: normal rows 0.4-0.8, other distributions below 1.1 (test_rows_of_other_distributions in test_f32_tensor_gpu.py; with one step of a float
// as the factor of Y and of the scale up to 2.6).  Sums that lose nothing (small whole numbers) get up to 1.5e-7 of a score too much.
template <int D>
struct Loss {
    static constexpr float kLog2eUp = kLog2e + (D == 64 ? 1 : 2) * 0x1p-23f;                           // log2 e, times 1 + kScore
    static constexpr float kScore = static_cast<float>(kLog2eUp / 1.4426950408889634 - 1.0);           // 6.9e-8, 1.5e-7
    static constexpr float kGrad = D == 64 ? 4e-8f : 9e-8f;
    static constexpr float kOut = 2.5e-8f, kGradOut = 7e-8f;
};

enum Use { kForward, kDv, kDq, kDk };

template <int D, int USE>
struct Plan {
    static constexpr bool kPair = USE == kDq || USE == kDk;            // two score products
    static constexpr int kPlane = kCols * D * 2;                       // one term of a streamed block
    static constexpr int kBlock = 3 * kPlane;
    static constexpr int kSmemTerms = kPair && D == 128 ? 2 : 0;       // terms of A2 in shared memory: TMEM holds one beside the rest
    static constexpr int kTmemTerms = kPair ? 3 - kSmemTerms : 0;
    static constexpr int kSlots = kPair && D == 128 ? 1 : 2;           // score slots
    static constexpr int kRing = D == 64 ? 6 : kPair ? 3 : 4;          // streamed blocks in shared memory
    static constexpr int kSlotCols = kPair ? 128 : 96;
    static constexpr int kColA2 = 3 * D / 2, kColX = kColA2 + kTmemTerms * D / 2, kColSum = kColX + kSlots * kSlotCols;
    static_assert(kColSum + D <= 512, "tensor memory");
    static constexpr int kA2Plane = kRows * D * 2;
    // A1 and A2 pass through the end of the ring; the blocks before that are free from the start
    static constexpr int kStage = kRows * D * 4, kStageA1 = kRing * kBlock - kStage, kFreeBlocks = (kRing * kBlock - (kPair ? 2 : 1) * kStage) / kBlock;
};

struct __align__(16) Shared {
    uint64_t block_full[6], block_empty[6];
    uint64_t x_full[2], y_full[2], w_full[2];
    uint64_t sum_full, sum_empty, alpha_full[4], rows_ready, drained;
    uint32_t tmem_base;
    int abort_flag, outside;
    float alpha[4][kRows];          // forward: what a block scales the sum by
    float total[kRows];             // forward: sum of the weights
    alignas(16) float of_queries[4][2][kCols];  // dV, dK: LSE and Di of the block's queries, a copy per warp
};
template <int D, int USE> constexpr int dynamic_smem() { return Plan<D, USE>::kRing * Plan<D, USE>::kBlock + Plan<D, USE>::kSmemTerms * Plan<D, USE>::kA2Plane + 1024; }      // 1 KB to align the swizzled tiles
static_assert(dynamic_smem<128, kDq>() + sizeof(Shared) <= 227 * 1024, "shared memory");

// One (batch, head) of a call as the kernel body sees it.
struct Job {
    const float *a1, *a2, *b1, *b2;            // row 0 of each operand
    const unsigned char *terms1, *terms2;      // terms of B1 and B2, block 0
    const int *marks1, *marks2;                // per block: a value out of range
    long long ld_a1, ld_a2, ld_b1, ld_b2;
    int row0, rows;                            // rows row0 .. min(row0 + 128, rows) are computed
    int col0, cols;                            // columns col0 .. cols are walked (col0 a multiple of 64)
    int causal, shift;                         // forward, dQ: column c is visible to row r iff c <= r + shift; dV, dK: iff r <= c
    float scale;
    const float *lse, *delta;                  // of the queries (backward)
    const float2* rope;                        // [rows, D/2] for A1, or null
    float* out;
    long long ld_out;
    float* lse_out;                            // forward, may be null
};

template <int USE>
__device__ __forceinline__ bool visible(const Job& j, int r, int c) {
    return c < j.cols && (USE == kForward || r < j.rows) && (!j.causal || (USE == kForward || USE == kDq ? c <= r + j.shift : r <= c));
}

// a, b = sum of three bf16 terms each (packed, a in the low half); chk turns NaN when one of them is not finite in bf16
__device__ __forceinline__ void split3(float a, float b, uint32_t& t0, uint32_t& t1, uint32_t& t2, float2& chk) {
    using E = Elem<__nv_bfloat16>;
    const float2 minus = make_float2(-1.f, -1.f), zero = make_float2(0.f, 0.f);
    t0 = E::pack2(a, b);
    const float2 f0 = E::unpack2(t0);
    chk = __ffma2_rn(f0, zero, chk);
    const float2 r1 = __ffma2_rn(f0, minus, make_float2(a, b));
    t1 = E::pack2(r1.x, r1.y);
    const float2 r2 = __ffma2_rn(E::unpack2(t1), minus, r1);
    t2 = E::pack2(r2.x, r2.y);
}
// volatile: the loads stay where the pipeline puts them, ahead of the waits and conversions before their use
__device__ __forceinline__ float4 load4(const float* p, bool valid) {
    float4 x;
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %5, 0;\n\tmov.b32 %0, 0;\n\tmov.b32 %1, 0;\n\tmov.b32 %2, 0;\n\tmov.b32 %3, 0;\n\t"
        "@p ld.global.nc.v4.f32 {%0, %1, %2, %3}, [%4];\n\t}"
        : "=&f"(x.x), "=&f"(x.y), "=&f"(x.z), "=&f"(x.w) : "l"(p), "r"(static_cast<int>(valid)));
    return x;
}
// The least magnitude but zero that has been met, as twice its bits less one: zero, of either sign, becomes the largest.
__device__ __forceinline__ uint32_t doubled(float x) { return 2 * __float_as_uint(x) - 1; }
__device__ __forceinline__ uint32_t least_of(uint32_t least, float4 x) { return min(least, min(min(doubled(x.x), doubled(x.y)), min(doubled(x.z), doubled(x.w)))); }
__device__ __forceinline__ bool too_small(uint32_t least) { return least < doubled(kLeast); }
// e^(x (1 + kScore)), x finite, with the rounding of the exponent x log2 e made up for
template <int D>
__device__ __forceinline__ float2 exp_pair(float2 x) {
    const float2 t = __fmul2_rn(x, make_float2(kLog2e, kLog2e)), lost = __ffma2_rn(x, make_float2(Loss<D>::kLog2eUp, Loss<D>::kLog2eUp), make_float2(-t.x, -t.y));
    const float2 y = make_float2(fast_exp2(t.x), fast_exp2(t.y));
    return __ffma2_rn(y, __fmul2_rn(lost, make_float2(kLn2, kLn2)), y);
}
__device__ __forceinline__ bool not_zero(float2 chk) { return !(chk.x + chk.y == 0.f); }

__device__ __forceinline__ void store_shared(uint32_t at, const uint32_t* x) { asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(at), "r"(x[0]), "r"(x[1]), "r"(x[2]), "r"(x[3])); }

__device__ __forceinline__ float4 rotated(float4 x, const float2* t) {
    const float2 c0 = t[0], c1 = t[1];
    return make_float4(__fsub_rn(__fmul_rn(x.x, c0.x), __fmul_rn(x.y, c0.y)), __fadd_rn(__fmul_rn(x.x, c0.y), __fmul_rn(x.y, c0.x)),
                       __fsub_rn(__fmul_rn(x.z, c1.x), __fmul_rn(x.w, c1.y)), __fadd_rn(__fmul_rn(x.z, c1.y), __fmul_rn(x.w, c1.x)));
}

// v[i], i < 32, of every lane -> lane i has the sum over the lanes of v[i]: halves of the values are exchanged, 31 shuffles in place of 160.
__device__ __forceinline__ float sum_across(float (&v)[32]) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
        for (int i = 0; i < o; ++i) {
            const bool upper = lane & o;
            const float send = upper ? v[i] : v[i + o], keep = upper ? v[i + o] : v[i];
            v[i] = keep + __shfl_xor_sync(0xFFFFFFFFu, send, o);
        }
    return v[0];
}

// The same rows by plain loops, masked columns left out: a warp takes four rows and eight columns at a time, for the products with a lane per D / 32
// dimensions, for the weights with a lane per (row, column).  Bound by shuffles, about 60 of them (forward) to 130 (dQ, dK) per 32 weights, on ten warps
// of an SM.  One NaN in every head of V, forward / backward: 2 x 8 x 512 x 64 360 / 406 us, 2 x 16 x 1999 x 128 3460 / 8360 (each value summed over the
// lanes by itself, four columns at a time: 910 / 1185, 7330 / 29250; the CUDA-core kernels, which have no such case: 87 / 160, 1150 / 3120).
template <int D, int USE>
__device__ __noinline__ void plain_rows(const Job j) {
    constexpr int V = D / 32, R = 4, C = 8;
    constexpr bool kPair = Plan<D, USE>::kPair;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, mine_q = lane / C, mine_k = lane % C;
    for (int r0 = j.row0 + warp * R; r0 < min(j.row0 + kRows, j.rows); r0 += kThreads / 32 * R) {
        float a1[R][V], a2[R][V], acc[R][V], m = -INFINITY, l = 0.f;     // m, l: of row mine_q
#pragma unroll
        for (int q = 0; q < R; ++q) {
            const int r = min(r0 + q, j.rows - 1);
#pragma unroll
            for (int i = 0; i < V; ++i) {
                const int d = lane + 32 * i;
                a1[q][i] = j.a1[r * j.ld_a1 + d];
                a2[q][i] = kPair ? j.a2[r * j.ld_a2 + d] : 0.f;
                acc[q][i] = 0.f;
                if (USE == kForward && j.rope != nullptr) {
                    const float2 cs = j.rope[static_cast<long long>(r) * (D / 2) + d / 2];
                    const float other = __shfl_xor_sync(0xFFFFFFFFu, a1[q][i], 1);
                    a1[q][i] = lane & 1 ? __fadd_rn(__fmul_rn(other, cs.y), __fmul_rn(a1[q][i], cs.x)) : __fsub_rn(__fmul_rn(a1[q][i], cs.x), __fmul_rn(other, cs.y));
                }
            }
        }
        const int row = r0 + mine_q;
#pragma unroll 1
        for (int c0 = j.col0; c0 < j.cols; c0 += C) {
            float b1[C][V], b2[C][V];
#pragma unroll
            for (int k = 0; k < C; ++k) {
                const long long c = min(c0 + k, j.cols - 1);
#pragma unroll
                for (int i = 0; i < V; ++i) {
                    b1[k][i] = j.b1[c * j.ld_b1 + lane + 32 * i];
                    b2[k][i] = j.b2[c * j.ld_b2 + lane + 32 * i];
                }
            }
            auto product = [&](const float (&a)[R][V], const float (&b)[C][V]) {
                float v[R * C];
#pragma unroll
                for (int q = 0; q < R; ++q)
#pragma unroll
                    for (int k = 0; k < C; ++k) {
                        v[q * C + k] = 0.f;
#pragma unroll
                        for (int i = 0; i < V; ++i) v[q * C + k] = fmaf(a[q][i], b[k][i], v[q * C + k]);
                    }
                return sum_across(v);
            };
            const float s = product(a1, b1), y = kPair ? product(a2, b2) : 0.f;
            const int col = c0 + mine_k, at = USE == kDq ? row : col;
            const bool seen = row < j.rows && visible<USE>(j, row, col);
            float w = 0.f;
            if constexpr (USE == kForward) {
                float top = seen ? s * j.scale : -INFINITY;
                const float x = top;
#pragma unroll
                for (int o = C / 2; o > 0; o >>= 1) top = fmaxf(top, __shfl_xor_sync(0xFFFFFFFFu, top, o));
                top = fmaxf(top, m);
                const float ref = top == -INFINITY ? 0.f : top, alpha = expf(m - ref);
                if (seen) w = expf(x - ref);
                float sum = w;
#pragma unroll
                for (int o = C / 2; o > 0; o >>= 1) sum += __shfl_xor_sync(0xFFFFFFFFu, sum, o);
                l = fmaf(l, alpha, sum);
                m = top;
#pragma unroll
                for (int q = 0; q < R; ++q) {
                    const float f = __shfl_sync(0xFFFFFFFFu, alpha, q * C);
#pragma unroll
                    for (int i = 0; i < V; ++i) acc[q][i] *= f;
                }
            } else if (seen) {
                w = expf(s * j.scale - j.lse[at]);
                if (kPair) w *= y - __ldcg(j.delta + at);
            }
            const unsigned all = __ballot_sync(0xFFFFFFFFu, seen);
            if (all == ~0u) {
#pragma unroll
                for (int q = 0; q < R; ++q)
#pragma unroll
                    for (int k = 0; k < C; ++k) {
                        const float f = __shfl_sync(0xFFFFFFFFu, w, q * C + k);
#pragma unroll
                        for (int i = 0; i < V; ++i) acc[q][i] = fmaf(f, kPair ? b1[k][i] : b2[k][i], acc[q][i]);
                    }
            } else {                                                     // (a weight of 0 times an infinity would be seen)
#pragma unroll 1
                for (int k = 0; k < min(C, j.cols - c0); ++k) {
                    const float* from = (kPair ? j.b1 + (c0 + k) * j.ld_b1 : j.b2 + (c0 + k) * j.ld_b2) + lane;
                    float b[V];
#pragma unroll
                    for (int i = 0; i < V; ++i) b[i] = from[32 * i];
#pragma unroll
                    for (int q = 0; q < R; ++q) {
                        const float f = __shfl_sync(0xFFFFFFFFu, w, q * C + k);
                        if (all >> (q * C + k) & 1)
#pragma unroll
                            for (int i = 0; i < V; ++i) acc[q][i] = fmaf(f, b[i], acc[q][i]);
                    }
                }
            }
        }
#pragma unroll
        for (int q = 0; q < R; ++q) {
            const int r = r0 + q;
            const float f = USE == kForward ? 1.0f / __shfl_sync(0xFFFFFFFFu, l, q * C) : USE == kDv ? 1.f : j.scale;
            if (r < j.rows)
#pragma unroll
                for (int i = 0; i < V; ++i) j.out[r * j.ld_out + lane + 32 * i] = acc[q][i] * f;
        }
        if (USE == kForward && j.lse_out != nullptr && mine_k == 0 && row < j.rows) j.lse_out[row] = m + logf(l);
    }
}

// every thread of the CTA, from wherever its role ends
__device__ __forceinline__ void roles_end() { asm volatile("bar.sync 1, %0;" ::"n"(kThreads) : "memory"); }

// The CTA's rows of A1 or A2 on their way into shared memory as they are: [128][D] floats, 16-byte word c of row r at word c ^ (r & 7).
// Rows at or after `rows` become zeros.  Warps 0-7.
template <int D>
__device__ __forceinline__ void fetch_rows(const float* src, long long ld, int row0, int rows, uint32_t stage) {
    for (int i = threadIdx.x; i < kRows * (D / 4); i += 256) {
        const int r = i / (D / 4), c = i % (D / 4), n = row0 + r < rows ? 16 : 0;
        const float* at = n ? src + (row0 + r) * ld + 4 * c : src;
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(stage + r * (D * 4) + ((c ^ (r & 7)) << 4)), "l"(at), "r"(n) : "memory");
    }
}

// From there into TMEM, a row per thread of warps 0-3 (first half of the columns) and 4-7; all three terms, or (A2, where TMEM has no room)
// the first, and the others into shared memory.  True if a value is out of range.
template <int D, int TMEM_TERMS>
__device__ __forceinline__ bool resident(const float2* rope, int row0, int rows, uint32_t stage, uint32_t col, uint32_t smem) {
    const int warp = threadIdx.x >> 5, half = warp >> 2, r = threadIdx.x & 127, row = row0 + r;
    const uint32_t lanes = static_cast<uint32_t>((warp & 3) * 32) << 16;
    float2 chk = make_float2(0.f, 0.f);
    uint32_t least = ~0u;
#pragma unroll 2
    for (int c = half * (D / 2); c < (half + 1) * (D / 2); c += 16) {
        const uint32_t at = lanes + col + c / 2;
        uint32_t t0[8], t1[8], t2[8];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            float4 v;
            asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(stage + r * (D * 4) + (((c / 4 + i) ^ (r & 7)) << 4)));
            if (rope != nullptr && row < rows) v = rotated(v, rope + static_cast<long long>(row) * (D / 2) + c / 2 + 2 * i);
            least = least_of(least, v);
            split3(v.x, v.y, t0[2 * i], t1[2 * i], t2[2 * i], chk);
            split3(v.z, v.w, t0[2 * i + 1], t1[2 * i + 1], t2[2 * i + 1], chk);
        }
        tmem_st8(at, t0);
        if (TMEM_TERMS == 3) {
            tmem_st8(at + D / 2, t1);
            tmem_st8(at + D, t2);
        } else {
            const uint32_t dst = smem + (c >> 6) * (kRows * 128) + r * 128;
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                const int at16 = ((((c & 63) >> 3) + i) ^ (r & 7)) << 4;
                store_shared(dst + at16, t1 + 4 * i);
                store_shared(dst + kRows * D * 2 + at16, t2 + 4 * i);
            }
        }
    }
    return too_small(least) || not_zero(chk);
}

// the warp's arrival, after what its lanes have done
__device__ __forceinline__ void warp_arrive(uint64_t* bar) {
    __syncwarp();
    if ((threadIdx.x & 31) == 0) mbar_arrive(bar);
}

template <int D, int USE>
__device__ __forceinline__ void attend(const Job& j, unsigned char* tiles, Shared& sh, int* status) {
    using P = Plan<D, USE>;
    constexpr bool kPair = P::kPair;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int n = (j.cols - j.col0 + kCols - 1) / kCols;                 // blocks, at least one
    unsigned char* a2_smem = tiles + P::kRing * P::kBlock;
    constexpr uint32_t tmem = 0;                 // all 512 columns are this CTA's
    const WaitCtx ctx{&sh.abort_flag, status};

    if (warp < 8) {
        // ---- A1 and A2 ----
        const uint32_t stage = smem_u32(tiles) + P::kStageA1;
        fetch_rows<D>(j.a1, j.ld_a1, j.row0, j.rows, stage);
        if constexpr (kPair) fetch_rows<D>(j.a2, j.ld_a2, j.row0, j.rows, stage - P::kStage);
        asm volatile("cp.async.wait_all;\n\tbar.sync 2, 256;" ::: "memory");
        bool outside = resident<D, 3>(USE == kForward ? j.rope : nullptr, j.row0, j.rows, stage, 0, 0);
        if constexpr (kPair) outside |= resident<D, P::kTmemTerms>(nullptr, j.row0, j.rows, stage - P::kStage, P::kColA2, smem_u32(a2_smem));
        if (outside) sh.outside = 1;
        tmem_st_wait();
        fence_proxy_async_smem();
        tc_fence_before();
        warp_arrive(&sh.rows_ready);
    }
    asm volatile("griddepcontrol.wait;" ::: "memory");      // the terms and Di are there (A1, A2 are inputs of the call)
    if (warp < 4) {
        // ---- weights of a block ----
        const int r = tid, row = j.row0 + r;
        const uint32_t lanes = static_cast<uint32_t>(warp * 32) << 16;
        const bool by_row = USE == kForward || USE == kDq;               // the queries are the rows
        float lse = 0.f, delta = 0.f;
        if (USE == kDq && row < j.rows) { lse = __ldg(j.lse + row); delta = __ldcg(j.delta + row); }
        float ahead[4] = {0.f, 0.f, 0.f, 0.f};                           // dV, dK: LSE and Di of two queries of the next block
        auto fetch = [&](int blk) {
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                const int c = j.col0 + blk * kCols + i * 32 + lane;
                if (c >= j.cols) ahead[i] = ahead[2 + i] = 0.f;
                else { ahead[i] = __ldg(j.lse + c); if (kPair) ahead[2 + i] = __ldcg(j.delta + c); }
            }
        };
        float (&of_queries)[2][kCols] = sh.of_queries[warp];
        if (!by_row) fetch(0);
        float m = -INFINITY, l = 0.f;
        // the row sees columns lo .. hi; every row of the tile sees some .. all
        int lo = 0, hi = j.cols, some = 0, all = j.cols;
        if (j.causal) {
            if (by_row) { hi = min(hi, row + j.shift + 1); all = min(all, j.row0 + j.shift + 1); }
            else { lo = row; some = j.row0 + kRows - 1; }
        }
        if (USE != kForward) {
            if (row >= j.rows) hi = lo;
            if (j.row0 + kRows > j.rows) all = 0;
        }
        const float2 scale = make_float2(j.scale, j.scale), lost = make_float2(j.scale * Loss<D>::kScore * kLog2e, j.scale * Loss<D>::kScore * kLog2e);
        float2 chk = make_float2(0.f, 0.f);
        bool ok = true;
        for (int blk = 0; blk < n; ++blk) {
            const int slot = blk % P::kSlots, turn = (blk / P::kSlots) & 1, c0 = j.col0 + blk * kCols;
            const uint32_t x = tmem + lanes + P::kColX + slot * P::kSlotCols;
            if (!by_row) {
                __syncwarp();                                            // the block before has been read
                of_queries[0][lane] = ahead[0]; of_queries[0][32 + lane] = ahead[1];
                of_queries[1][lane] = ahead[2]; of_queries[1][32 + lane] = ahead[3];
                __syncwarp();
                if (blk + 1 < n) fetch(blk + 1);
            }
            ok = mbar_wait_warp(&sh.x_full[slot], turn, ctx, 0x100);
            if (!ok) break;
            tc_fence_after();
            uint32_t u[2][32];
            tmem_ld32(x, u[0]);
            tmem_ld32(x + 32, u[1]);
            tmem_ld_wait();
            float* s = reinterpret_cast<float*>(u);
            // columns past the end, or masked ones: only the blocks at the edges have any
            const bool edge = c0 < some || c0 + kCols > all;
            if constexpr (USE == kForward) {
                float mx[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
                for (int i = 0; i < kCols; i += 2) {
                    const float2 x = __fmul2_rn(make_float2(s[i], s[i + 1]), scale);
                    s[i] = x.x; s[i + 1] = x.y;
                }
                if (edge)
#pragma unroll
                    for (int i = 0; i < kCols; ++i)
                        if (i < lo - c0 || i >= hi - c0) s[i] = -INFINITY;
#pragma unroll
                for (int i = 0; i < kCols; i += 2) mx[(i >> 1) & 3] = fmax3(mx[(i >> 1) & 3], s[i], s[i + 1]);
                const float top = fmaxf(m, fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3])));
                // (the first block holds a visible column: top is finite, or the rows are computed again)
                const float alpha = expf(m - top) * fmaf(fmaxf(m - top, -200.f), Loss<D>::kScore, 1.f);
#pragma unroll
                for (int i = 0; i < kCols; i += 2) {
                    const float2 x = __fadd2_rn(make_float2(s[i], s[i + 1]), make_float2(-top, -top)), w = exp_pair<D>(x);
                    s[i] = w.x; s[i + 1] = w.y;
                }
                if (edge)                                                // the weight itself: a score far enough below any top is not a number of 24 bits
#pragma unroll
                    for (int i = 0; i < kCols; ++i)
                        if (i < lo - c0 || i >= hi - c0) s[i] = 0.f;
                float2 sum[2] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
#pragma unroll
                for (int i = 0; i < kCols; i += 2) sum[(i >> 1) & 1] = __fadd2_rn(sum[(i >> 1) & 1], make_float2(s[i], s[i + 1]));
                l = fmaf(l, alpha, (sum[0].x + sum[0].y) + (sum[1].x + sum[1].y));
                m = top;
                sh.alpha[blk & 3][r] = alpha;
                warp_arrive(&sh.alpha_full[blk & 3]);
            } else {
#pragma unroll
                for (int i = 0; i < kCols; i += 4) {
                    float4 at = make_float4(lse, lse, lse, lse);
                    if (!by_row) at = *reinterpret_cast<const float4*>(&of_queries[0][i]);
                    const float2 s0 = make_float2(s[i], s[i + 1]), s1 = make_float2(s[i + 2], s[i + 3]);
                    const float2 log2e = make_float2(kLog2e, kLog2e);
                    const float2 t0 = __ffma2_rn(__ffma2_rn(s0, scale, make_float2(-at.x, -at.y)), log2e, __fmul2_rn(s0, lost));
                    const float2 t1 = __ffma2_rn(__ffma2_rn(s1, scale, make_float2(-at.z, -at.w)), log2e, __fmul2_rn(s1, lost));
                    s[i] = fast_exp2(t0.x); s[i + 1] = fast_exp2(t0.y); s[i + 2] = fast_exp2(t1.x); s[i + 3] = fast_exp2(t1.y);
                }
                if (edge)
#pragma unroll
                    for (int i = 0; i < kCols; ++i)
                        if (i < lo - c0 || i >= hi - c0) s[i] = 0.f;
            }
            if constexpr (kPair) {
                ok = mbar_wait_warp(&sh.y_full[slot], turn, ctx, 0x110);
                if (!ok) break;
                tc_fence_after();
            }
#pragma unroll
            for (int h = 0; h < 4; ++h) {
                float* w = s + h * 16;
                if constexpr (kPair) {
                    uint32_t y[16];
                    tmem_ld16(x + 64 + h * 16, y);
                    tmem_ld_wait();
#pragma unroll
                    for (int i = 0; i < 16; i += 4) {
                        float4 at = make_float4(delta, delta, delta, delta);
                        if (!by_row) at = *reinterpret_cast<const float4*>(&of_queries[1][h * 16 + i]);
                        const float2 y0 = make_float2(__uint_as_float(y[i]), __uint_as_float(y[i + 1])), y1 = make_float2(__uint_as_float(y[i + 2]), __uint_as_float(y[i + 3]));
                        const float2 lost = make_float2(Loss<D>::kGrad, Loss<D>::kGrad);
                        const float2 w0 = __fmul2_rn(make_float2(w[i], w[i + 1]), __ffma2_rn(y0, lost, __fadd2_rn(y0, make_float2(-at.x, -at.y))));
                        const float2 w1 = __fmul2_rn(make_float2(w[i + 2], w[i + 3]), __ffma2_rn(y1, lost, __fadd2_rn(y1, make_float2(-at.z, -at.w))));
                        w[i] = w0.x; w[i + 1] = w0.y; w[i + 2] = w1.x; w[i + 3] = w1.y;
                    }
                }
                uint32_t t0[8], t1[8], t2[8];
#pragma unroll
                for (int i = 0; i < 8; ++i) split3(w[2 * i], w[2 * i + 1], t0[i], t1[i], t2[i], chk);
                // (the third term goes where this quarter of Y, or one before it, has been read)
                tmem_st8(x + h * 8, t0);
                tmem_st8(x + 32 + h * 8, t1);
                tmem_st8(x + 64 + h * 8, t2);
            }
            tmem_st_wait();
            tc_fence_before();
            warp_arrive(&sh.w_full[slot]);
        }
        if (not_zero(chk) || (USE == kForward && !(l < INFINITY))) sh.outside = 1;
        if (USE == kForward) sh.total[r] = l;
        roles_end();
        if (USE == kForward && !sh.outside && j.lse_out != nullptr && row < j.rows) {
            const float d = m * Loss<D>::kScore;                         // within the logarithm while that is small: one rounding less
            j.lse_out[row] = m + (fabsf(d) < 1e-4f ? logf(fmaf(l, d, l)) : d + logf(l));
        }
    } else if (warp < kLoadWarp) {
        // ---- the sum ----
        const int r = tid & 127;
        float2 acc[D / 2];
#pragma unroll
        for (int i = 0; i < D / 2; ++i) acc[i] = make_float2(0.f, 0.f);
        const uint32_t sum = tmem + (static_cast<uint32_t>((warp & 3) * 32) << 16) + P::kColSum;
        bool ok = true;
        for (int blk = 0; blk < n; ++blk) {
            float2 alpha = make_float2(1.f, 1.f);
            if constexpr (USE == kForward) {
                ok = mbar_wait_warp(&sh.alpha_full[blk & 3], (blk >> 2) & 1, ctx, 0x200);
                if (!ok) break;
                alpha.x = alpha.y = sh.alpha[blk & 3][r];
            }
            ok = mbar_wait_warp(&sh.sum_full, blk & 1, ctx, 0x210);
            if (!ok) break;
            tc_fence_after();
#pragma unroll
            for (int h = 0; h < D / 16; ++h) {
                uint32_t o[16];
                tmem_ld16(sum + h * 16, o);
                tmem_ld_wait();
                if (h == D / 16 - 1) { tc_fence_before(); warp_arrive(&sh.sum_empty); }
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const float2 x = make_float2(__uint_as_float(o[2 * i]), __uint_as_float(o[2 * i + 1]));
                    acc[h * 8 + i] = USE == kForward ? __ffma2_rn(acc[h * 8 + i], alpha, x) : __fadd2_rn(acc[h * 8 + i], x);
                }
            }
        }
        roles_end();
        if (!sh.outside) {
            const float f = USE == kForward ? 1.0f / sh.total[r] : USE == kDv ? 1.f : j.scale;
            // through the ring, which is free now: a warp turns its 32 rows into stores of whole rows
            const uint32_t own = smem_u32(tiles) + (warp - 4) * (32 * D * 4);
#pragma unroll
            for (int i = 0; i < D / 4; ++i) {
                float v[4] = {acc[2 * i].x * f, acc[2 * i].y * f, acc[2 * i + 1].x * f, acc[2 * i + 1].y * f};
#pragma unroll
                for (int e = 0; e < 4; ++e) v[e] = fmaf(v[e], USE == kForward ? Loss<D>::kOut : Loss<D>::kGradOut, v[e]);
                store_shared(own + lane * (D * 4) + ((i ^ (lane & 7)) << 4), reinterpret_cast<const uint32_t*>(v));
            }
            __syncwarp();
            constexpr int kLanes = D / 4, kAtOnce = 32 / kLanes;
            const int c = lane % kLanes;
#pragma unroll 8
            for (int i = lane / kLanes; i < 32; i += kAtOnce) {
                const int to = j.row0 + (warp & 3) * 32 + i;
                float4 v;
                asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(own + i * (D * 4) + ((c ^ (i & 7)) << 4)));
                if (to < j.rows) *reinterpret_cast<float4*>(j.out + to * j.ld_out + 4 * c) = v;
            }
        }
    } else if (warp == kLoadWarp) {
        // ---- B1 and B2, in the order in which the products need them ----
        // Items 2 x, 2 x + 1 of the ring: pairs take B1 and B2 of one block after the other; otherwise B1 runs one block ahead.
        const int block0 = j.col0 / kCols;
        int marked = 0;
        for (int i = lane; i < n; i += 32) marked |= __ldcg(j.marks1 + block0 + i) | __ldcg(j.marks2 + block0 + i);
        if (marked) sh.outside = 1;
        if (lane == 0) {
            bool ok = true;
            for (int t = 0; t < 2 * n && ok; ++t) {
                const int slot = t % P::kRing, at = t >> 1, odd = t & 1;
                const bool second = kPair ? odd : odd ? at + 1 == n : at > 0;
                const int blk = kPair ? at : odd ? min(at + 1, n - 1) : max(at - 1, 0);
                if (t == P::kFreeBlocks) {                                       // A1 and A2 have left the ring
                    ok = mbar_wait(&sh.rows_ready, 0, ctx, 0x310);
                    fence_proxy_async_smem();
                }
                if (t >= P::kRing && ok) ok = mbar_wait(&sh.block_empty[slot], (t / P::kRing - 1) & 1, ctx, 0x300);
                if (!ok) break;
                mbar_arrive_expect_tx(&sh.block_full[slot], P::kBlock);
                bulk_load(tiles + slot * P::kBlock, (second ? j.terms2 : j.terms1) + static_cast<long long>(block0 + blk) * P::kBlock, P::kBlock, &sh.block_full[slot]);
            }
        }
        __syncwarp();
        roles_end();
    } else {
        // ---- products ----
        {
            // The whole warp walks the blocks and one lane issues: addresses and descriptors stay in uniform registers.
            constexpr uint32_t idesc_x = make_idesc_f16(Elem<__nv_bfloat16>::kFormat, 0, 0, kRows, kCols);
            constexpr uint32_t idesc_w = make_idesc_f16(Elem<__nv_bfloat16>::kFormat, 0, 1, kRows, D);
            // (term of A, term of B), smallest products first
            constexpr int kTermA[6] = {1, 0, 2, 0, 1, 0}, kTermB[6] = {1, 2, 0, 1, 0, 0};
            const bool leader = elect_one();
            const uint64_t by_k = make_smem_desc_sw128(smem_u32(tiles), 16, 1024);                    // a block as rows x head dimension
            const uint64_t by_row = make_smem_desc_sw128(smem_u32(tiles), kCols * 128, 1024);         // MN-major: 16 of its rows are 2048 bytes
            const uint64_t a2 = make_smem_desc_sw128(smem_u32(a2_smem), 16, 1024);
            bool ok = mbar_wait_warp(&sh.rows_ready, 0, ctx, 0x400);
            tc_fence_after();
            auto item = [&](bool second, int blk) {
                if (kPair) return 2 * blk + second;
                if (!second) return blk == 0 ? 0 : 2 * blk - 1;
                return blk + 1 < n ? 2 * blk + 2 : 2 * n - 1;
            };
            auto arrived = [&](int t, int where) {
                if (ok) ok = mbar_wait_warp(&sh.block_full[t % P::kRing], (t / P::kRing) & 1, ctx, where);
                if (ok) tc_fence_after();
                return ok;
            };
            auto product = [&](uint32_t d, uint32_t a_col, bool a_smem, int t) {       // d = A B^T over the head dimension
                const uint64_t b = by_k + (t % P::kRing) * (P::kBlock >> 4);
                if (leader)
#pragma unroll
                    for (int q = 0; q < 6; ++q)
#pragma unroll
                        for (int kk = 0; kk < D / 16; ++kk) {
                            const uint64_t bd = b + ((kTermB[q] * P::kPlane + (kk >> 2) * (kCols * 128) + (kk & 3) * 32) >> 4);
                            const uint32_t add = q > 0 || kk > 0;
                            if (a_smem && P::kSmemTerms > 0 && kTermA[q] > 0)
                                umma_ss(d, a2 + (((kTermA[q] - 1) * P::kA2Plane + (kk >> 2) * (kRows * 128) + (kk & 3) * 32) >> 4), bd, idesc_x, add);
                            else umma_ts(d, a_col + kTermA[q] * (D / 2) + kk * 8, bd, idesc_x, add);
                        }
            };
            auto commit = [&](uint64_t* bar) { if (leader) umma_commit(bar); };
            auto scores = [&](int blk) {
                const int slot = blk % P::kSlots, t1 = item(false, blk);
                const uint32_t x = tmem + P::kColX + slot * P::kSlotCols;
                if (!arrived(t1, 0x410)) return;
                product(x, tmem, false, t1);
                commit(&sh.x_full[slot]);
                if constexpr (kPair) {
                    const int t2 = item(true, blk);
                    if (!arrived(t2, 0x420)) return;
                    product(x + 64, tmem + P::kColA2, true, t2);
                    commit(&sh.y_full[slot]);
                    commit(&sh.block_empty[t2 % P::kRing]);
                } else commit(&sh.block_empty[t1 % P::kRing]);
            };
            if (ok && P::kSlots == 2) scores(0);
            for (int blk = 0; blk < n && ok; ++blk) {
                if (P::kSlots == 1) scores(blk);
                else if (blk + 1 < n) scores(blk + 1);
                const int slot = blk % P::kSlots, t = item(!kPair, blk);
                if (!arrived(t, 0x430)) break;
                ok = mbar_wait_warp(&sh.w_full[slot], (blk / P::kSlots) & 1, ctx, 0x440);
                if (ok && blk > 0) ok = mbar_wait_warp(&sh.sum_empty, (blk - 1) & 1, ctx, 0x450);
                if (!ok) break;
                tc_fence_after();
                const uint32_t w = tmem + P::kColX + slot * P::kSlotCols;
                const uint64_t b = by_row + (t % P::kRing) * (P::kBlock >> 4);
                if (leader)
#pragma unroll
                    for (int q = 0; q < 6; ++q)
#pragma unroll
                        for (int kk = 0; kk < kCols / 16; ++kk)
                            umma_ts(tmem + P::kColSum, w + kTermA[q] * (kCols / 2) + kk * 8, b + ((kTermB[q] * P::kPlane + kk * 2048) >> 4), idesc_w, q > 0 || kk > 0);
                commit(&sh.sum_full);
                commit(&sh.block_empty[t % P::kRing]);
            }
            // everything issued has to retire before TMEM is released
            commit(&sh.drained);
            mbar_wait_warp(&sh.drained, 0, ctx, 0x460);
        }
        __syncwarp();
        roles_end();
    }
    abort_linger(&sh.abort_flag);
    if (sh.outside && !sh.abort_flag) plain_rows<D, USE>(j);
}

__device__ __forceinline__ unsigned char* aligned_tiles(unsigned char* raw) {
    return reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(raw) + 1023) & ~uintptr_t(1023));
}

// barriers and tensor memory; every thread of the CTA
__device__ __forceinline__ void begin(Shared& sh) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (warp == kIssueWarp) {
        if (lane == 0) {
            for (int i = 0; i < 6; ++i) { mbar_init(&sh.block_full[i], 1); mbar_init(&sh.block_empty[i], 1); }
            for (int i = 0; i < 2; ++i) { mbar_init(&sh.x_full[i], 1); mbar_init(&sh.y_full[i], 1); mbar_init(&sh.w_full[i], 4); }
            for (int i = 0; i < 4; ++i) mbar_init(&sh.alpha_full[i], 4);
            mbar_init(&sh.sum_full, 1); mbar_init(&sh.sum_empty, 4); mbar_init(&sh.rows_ready, 8); mbar_init(&sh.drained, 1);
            sh.abort_flag = sh.outside = 0;
            mbar_fence_init();
        }
        __syncwarp();
        tmem_alloc(&sh.tmem_base, 512);
        tmem_relinquish();
        tc_fence_before();
    }
    __syncthreads();
    tc_fence_after();
}
__device__ __forceinline__ void end(Shared& sh) {
    tc_fence_before();
    __syncthreads();
    if ((threadIdx.x >> 5) == kIssueWarp) {
        tc_fence_after();
        tmem_dealloc(sh.tmem_base, 512);
    }
}

// ---- the terms of the streamed operands ----
struct SplitTensor {
    const float* src;                          // row 0 of (batch 0, head 0)
    long long sb, sh, ss;
    unsigned char* terms;                      // [heads][blocks][3][D / 64][64 rows][128 bytes], swizzled
    int* marks;                                // [heads][blocks]
};
struct SplitParams {
    SplitTensor t[4];
    int rows, heads_per_batch, first_head, blocks;
    const float* out;                          // backward: O, with which tensor 3 (dO) gives Di = rowsum(dO O)
    float* delta;
};

// grid (blocks of 64 rows, heads, tensors).  Bound by memory: 4 bytes read and 6 written per value.
template <int D>
__global__ void __launch_bounds__(256)
split_blocks_kernel(const __grid_constant__ SplitParams p) {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    const SplitTensor& t = p.t[blockIdx.z];
    const int head = p.first_head + blockIdx.y, row0 = blockIdx.x * kCols;
    const float* src = t.src + head / p.heads_per_batch * t.sb + head % p.heads_per_batch * t.sh;
    const long long block = static_cast<long long>(blockIdx.y) * p.blocks + blockIdx.x;
    unsigned char* dst = t.terms + block * (3 * kCols * D * 2);
    float2 chk = make_float2(0.f, 0.f);
    uint32_t least = ~0u;
    constexpr int kLanes = D / 8;              // threads of a row
#pragma unroll
    for (int i = 0; i < kCols * kLanes / 256; ++i) {
        const int at = threadIdx.x + i * 256, r = at / kLanes, c = at % kLanes * 8, row = row0 + r;
        const float4 x = load4(src + row * t.ss + c, row < p.rows), y = load4(src + row * t.ss + c + 4, row < p.rows);
        least = least_of(least_of(least, x), y);
        uint4 t0, t1, t2;
        split3(x.x, x.y, t0.x, t1.x, t2.x, chk);
        split3(x.z, x.w, t0.y, t1.y, t2.y, chk);
        split3(y.x, y.y, t0.z, t1.z, t2.z, chk);
        split3(y.z, y.w, t0.w, t1.w, t2.w, chk);
        unsigned char* to = dst + (c >> 6) * (kCols * 128) + r * 128 + ((((c & 63) >> 3) ^ (r & 7)) << 4);
        *reinterpret_cast<uint4*>(to) = t0;
        *reinterpret_cast<uint4*>(to + kCols * D * 2) = t1;
        *reinterpret_cast<uint4*>(to + 2 * kCols * D * 2) = t2;
        if (p.out != nullptr && blockIdx.z == 3) {
            const long long flat = static_cast<long long>(head) * p.rows + row;
            const float4 u = load4(p.out + flat * D + c, row < p.rows), v = load4(p.out + flat * D + c + 4, row < p.rows);
            float d = fmaf(x.x, u.x, fmaf(x.y, u.y, fmaf(x.z, u.z, x.w * u.w))) + fmaf(y.x, v.x, fmaf(y.y, v.y, fmaf(y.z, v.z, y.w * v.w)));
#pragma unroll
            for (int o = kLanes / 2; o > 0; o >>= 1) d += __shfl_xor_sync(0xFFFFFFFFu, d, o);
            if (c == 0 && row < p.rows) p.delta[flat] = d;
        }
    }
    const int any = __syncthreads_or(too_small(least) || not_zero(chk));
    if (threadIdx.x == 0) t.marks[block] = any;
}

// The workspace of `heads` heads of `rows` rows: terms of each tensor, then their marks.
struct SplitLayout {
    int blocks;
    size_t terms_bytes, marks_bytes;           // of one tensor
    SplitLayout(int rows, int D, int heads) {
        blocks = (rows + kCols - 1) / kCols;
        terms_bytes = static_cast<size_t>(heads) * blocks * (3 * kCols * 2) * D;
        marks_bytes = (static_cast<size_t>(heads) * blocks * sizeof(int) + 255) / 256 * 256;
    }
};
// Heads whose terms and marks are in the workspace at a time: as many as one gigabyte holds, and at least one.
constexpr size_t kWorkspaceGoal = size_t{1} << 30;
int heads_at_a_time(int rows, int D, int heads, int tensors) {
    const SplitLayout one(rows, D, 1);
    size_t most = (kWorkspaceGoal - tensors * 256) / (tensors * (one.terms_bytes + one.blocks * sizeof(int)));      // (marks are rounded up to 256 bytes)
    if (most > 65535) most = 65535;            // the second dimension of a grid
    return most < 1 ? 1 : most < static_cast<size_t>(heads) ? static_cast<int>(most) : heads;
}
size_t split_bytes(int rows, int D, int heads, int tensors) {
    const SplitLayout l(rows, D, heads_at_a_time(rows, D, heads, tensors));
    return tensors * (l.terms_bytes + l.marks_bytes);
}

struct Split {                                 // where the terms of one launch are
    const unsigned char* terms[4];
    const int* marks[4];
    int blocks, first_head, heads;
};

// rows of the tile with the most visible columns first
template <int D>
__global__ void __launch_bounds__(kThreads, 1)
attention_f32_forward_kernel(const __grid_constant__ PrefillParams p, const __grid_constant__ Split w) {
    extern __shared__ unsigned char raw[];
    __shared__ Shared sh;
    begin(sh);
    const int group = p.Hq / p.Hkv, heads = w.heads * group, tiles = (p.T + kRows - 1) / kRows;
    const int at = tiles - 1 - blockIdx.x / heads, mine = blockIdx.x % heads, kv = mine / group;
    const int head = w.first_head + kv, b = head / p.Hkv, hkv = head % p.Hkv, h = hkv * group + mine % group;
    Job j{};
    j.a1 = static_cast<const float*>(p.q.ptr) + b * p.q.sb + h * p.q.sh; j.ld_a1 = p.q.ss;
    j.b1 = static_cast<const float*>(p.k.ptr) + b * p.k.sb + hkv * p.k.sh; j.ld_b1 = p.k.ss;
    j.b2 = static_cast<const float*>(p.v.ptr) + b * p.v.sb + hkv * p.v.sh; j.ld_b2 = p.v.ss;
    const long long block = static_cast<long long>(kv) * w.blocks;
    j.terms1 = w.terms[0] + block * (3 * kCols * D * 2); j.marks1 = w.marks[0] + block;
    j.terms2 = w.terms[1] + block * (3 * kCols * D * 2); j.marks2 = w.marks[1] + block;
    j.row0 = at * kRows; j.rows = p.T; j.col0 = 0;
    j.causal = p.causal; j.shift = p.start_pos;
    j.cols = p.causal ? min(p.Skv, p.start_pos + min(j.row0 + kRows, p.T)) : p.Skv;
    j.scale = p.scale; j.rope = p.q_rope_table;
    j.out = static_cast<float*>(p.o.ptr) + b * p.o.sb + h * p.o.sh; j.ld_out = p.o.ss;
    j.lse_out = p.lse != nullptr ? p.lse + (static_cast<long long>(b) * p.Hq + h) * p.T : nullptr;
    attend<D, kForward>(j, aligned_tiles(raw), sh, p.status);
    end(sh);
}

// dQ, dK and dV of a tile level for all heads, then the next level: dQ from the last query tile on, dK and dV from the first key tile
template <int D>
__global__ void __launch_bounds__(kThreads, 1)
attention_f32_backward_kernel(const __grid_constant__ AttnBwdParams p, const __grid_constant__ Split w) {
    extern __shared__ unsigned char raw[];
    __shared__ Shared sh;
    begin(sh);
    const int tiles = (p.N + kRows - 1) / kRows, level = blockIdx.x / (3 * w.heads), rest = blockIdx.x % (3 * w.heads), what = rest / w.heads, mine = rest % w.heads;
    const long long bh = w.first_head + mine, first = bh * p.N * D, block = static_cast<long long>(mine) * w.blocks;
    const float *q = p.q + first, *k = p.k + first, *v = p.v + first, *g = p.d_out + first;
    Job j{};
    j.ld_a1 = j.ld_a2 = j.ld_b1 = j.ld_b2 = j.ld_out = D;
    j.rows = j.cols = p.N;
    j.causal = p.causal; j.scale = p.scale;
    j.lse = p.lse + bh * p.N; j.delta = p.delta + bh * p.N;
    const int t1 = what == 0 ? 1 : 0, t2 = what == 0 ? 2 : 3;      // tensors of the workspace: Q, K, V, dO
    j.terms1 = w.terms[t1] + block * (3 * kCols * D * 2); j.marks1 = w.marks[t1] + block;
    j.terms2 = w.terms[t2] + block * (3 * kCols * D * 2); j.marks2 = w.marks[t2] + block;
    if (what == 0) {
        j.row0 = (tiles - 1 - level) * kRows;
        if (p.causal) j.cols = min(p.N, j.row0 + kRows);
        j.a1 = q; j.a2 = g; j.b1 = k; j.b2 = v; j.out = p.dq + first;
        attend<D, kDq>(j, aligned_tiles(raw), sh, p.status);
    } else {
        j.row0 = level * kRows;
        if (p.causal) j.col0 = j.row0;            // queries before the keys see none of them
        j.a1 = k; j.b1 = q; j.b2 = g;
        if (what == 1) {
            j.a2 = v; j.out = p.dk + first;
            attend<D, kDk>(j, aligned_tiles(raw), sh, p.status);
        } else {
            j.out = p.dv + first;
            attend<D, kDv>(j, aligned_tiles(raw), sh, p.status);
        }
    }
    end(sh);
}

// Raises a kernel's shared memory limit once per device ordinal and thread (the attribute belongs to the device's context).
template <typename Kernel>
int raise_smem(Kernel kernel, int bytes, bool* configured) {
    int dev = 0;
    VB200_CUDA_TRY(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64) return set_detail(VB200_ERR_NO_DEVICE, "device ordinal out of range");
    if (!configured[dev]) {
        VB200_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes));
        configured[dev] = true;
    }
    return VB200_OK;
}

// Splits `tensors` tensors of heads first .. first + heads, then launches the attention kernel behind it.
template <int D, typename Kernel, typename Params>
int run(cudaStream_t s, SplitParams& sp, unsigned char* workspace, int tensors, int heads, int tiles, Kernel kernel, int smem, const Params& p) {
    const int group = heads_at_a_time(sp.rows, D, heads, tensors);
    const SplitLayout l(sp.rows, D, group);
    Split w{};
    for (int i = 0; i < tensors; ++i) {
        w.terms[i] = sp.t[i].terms = workspace + i * l.terms_bytes;
        w.marks[i] = sp.t[i].marks = reinterpret_cast<int*>(workspace + tensors * l.terms_bytes + i * l.marks_bytes);
    }
    w.blocks = sp.blocks = l.blocks;
    for (int first = 0; first < heads; first += group) {
        w.first_head = sp.first_head = first;
        w.heads = heads - first < group ? heads - first : group;
        split_blocks_kernel<D><<<dim3(l.blocks, w.heads, tensors), 256, 0, s>>>(sp);
        note_launch();
        VB200_CUDA_TRY(cudaPeekAtLastError());
        if (int rc = launch_pdl(kernel, dim3(static_cast<unsigned>(tiles) * w.heads), dim3(kThreads), smem, s, p, w)) return rc;
    }
    return VB200_OK;
}

template <int D>
int forward_t(cudaStream_t s, const PrefillParams& p, unsigned char* workspace) {
    static thread_local bool configured[64] = {};
    constexpr int smem = dynamic_smem<D, kForward>();
    if (int rc = raise_smem(attention_f32_forward_kernel<D>, smem, configured)) return rc;
    SplitParams sp{};
    sp.t[0] = SplitTensor{static_cast<const float*>(p.k.ptr), p.k.sb, p.k.sh, p.k.ss, nullptr, nullptr};
    sp.t[1] = SplitTensor{static_cast<const float*>(p.v.ptr), p.v.sb, p.v.sh, p.v.ss, nullptr, nullptr};
    sp.rows = p.Skv; sp.heads_per_batch = p.Hkv;
    note_prefill_kernel("attention_f32_forward_kernel");
    return run<D>(s, sp, workspace, 2, p.B * p.Hkv, (p.T + kRows - 1) / kRows * (p.Hq / p.Hkv), attention_f32_forward_kernel<D>, smem, p);
}

template <int D>
int backward_t(cudaStream_t s, const AttnBwdParams& p, unsigned char* workspace) {
    static thread_local bool configured[64] = {};
    constexpr int smem = dynamic_smem<D, kDq>() > dynamic_smem<D, kDv>() ? dynamic_smem<D, kDq>() : dynamic_smem<D, kDv>();
    if (int rc = raise_smem(attention_f32_backward_kernel<D>, smem, configured)) return rc;
    SplitParams sp{};
    const float* src[4] = {p.q, p.k, p.v, p.d_out};
    for (int i = 0; i < 4; ++i) sp.t[i] = SplitTensor{src[i], static_cast<long long>(p.H) * p.N * D, static_cast<long long>(p.N) * D, D, nullptr, nullptr};
    sp.rows = p.N; sp.heads_per_batch = p.H;
    sp.out = p.out; sp.delta = p.delta;
    return run<D>(s, sp, workspace, 4, p.B * p.H, (p.N + kRows - 1) / kRows * 3, attention_f32_backward_kernel<D>, smem, p);
}

}  // namespace

size_t prefill_f32_split_bytes(int D, int kv_heads, int keys) { return split_bytes(keys, D, kv_heads, 2); }
size_t attention_bwd_f32_split_bytes(int D, int heads, int N) { return split_bytes(N, D, heads, 4); }

int launch_prefill_f32_sm100(cudaStream_t s, const PrefillParams& p, void* workspace) {
    unsigned char* ws = static_cast<unsigned char*>(workspace);
    return p.D == 64 ? forward_t<64>(s, p, ws) : forward_t<128>(s, p, ws);
}
int launch_attention_bwd_f32_sm100(cudaStream_t s, const AttnBwdParams& p, void* workspace) {
    unsigned char* ws = static_cast<unsigned char*>(workspace);
    return p.D == 64 ? backward_t<64>(s, p, ws) : backward_t<128>(s, p, ws);
}

}  // namespace vb200
