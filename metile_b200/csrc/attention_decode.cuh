// Decode attention (one query row per sequence and head) over an in-place KV cache, grouped-query
// aware, plus the rotary embedding + cache append that precedes it in a decoder block.
//
// Computes what the reference's kernels/attention.py:27-143 computes -- softmax(q.k * scale) @ v per
// (batch, query head), query head h reading KV head h / (Hq / Hkv) (:41-44), every load cast to fp32
// before it is multiplied (:58-62), fp32 accumulation, one rounding at the store -- behind the
// admission rule of metile/integrations/mlx_lm.py:3558-3573 (query length one, no mask, equal K/V
// shapes, head dim a multiple of 32).  The reference launches one threadgroup per (batch, QUERY head),
// so a KV head's keys and values are streamed once per query head of its group; here one CTA serves
// every query head of a KV head, so each cache byte is read once.
//
// Split over the KV range ("flash decoding"): CTA (s, b*Hkv + h) takes tokens [128 s, 128 s + 128) of
// one (sequence, KV head).  Its key and value tiles (35 KB each at head dim 128, rows padded by 16
// bytes) are copied to shared memory by 16-byte asynchronous copies issued before anything else, so
// the whole tile pair is in flight at once; the arithmetic runs on the tensor cores (see the kernel):
// scores K . Q^T with the KV head's query-head group as the N dimension, softmax on the score
// fragments in registers, values P . V with the probabilities split into two bf16 numbers; the CTA's
// partial (max, sum, O) goes to the caller's scratch and a second kernel merges the splits in split
// order.  The reference multiplies fp32 casts of the same bf16 inputs (:58-62); the products are
// exact either way, the sums are fp32, and the scale multiplies the fp32 score instead of the query.
// The split size is a constant, so a (sequence, head)'s bits depend on its own KV length only -- not
// on how many sequences share the launch.
//
// Bytes: K and V rows of the tokens in use, 2 * B * Hkv * N * D * 2; everything else is noise.
#pragma once

#include "common.cuh"
#include "ptx.cuh"

namespace mt {

constexpr int kAttnSplitTokens = 128;  // tokens per CTA: four groups of 32 lanes
constexpr int kAttnMaxGroup = 8;       // query heads per KV head

struct AttentionParams {
    const uint16_t* q;        // [B, Hq, D] bf16
    const uint16_t* k;        // [B, Hkv, capacity, D] bf16
    const uint16_t* v;
    const int* lengths;       // [B] tokens in use per sequence, or null: `tokens` for all
    float* partial;           // [B*Hkv, splits, G, D + 2] fp32 (caller scratch); unused when splits == 1
    uint16_t* out;            // [B, Hq, D] bf16
    int q_heads, kv_heads, capacity, tokens, splits;
    float scale;
};

constexpr int kAttnThreads = 256;
constexpr int kAttnRowPad = 8;  // bf16 elements: a tile row in shared memory is 16 bytes longer than in the cache

template <int kD>
constexpr int attention_smem_bytes() {
    return 2 * kAttnSplitTokens * (kD + kAttnRowPad) * 2;  // key tile + value tile
}

// Four 8x8 b16 matrices from shared memory into the fragment layout of mma.sync (lane l supplies the
// address of row l % 8 of matrix l / 8); `trans` delivers each matrix transposed.
__device__ __forceinline__ void ldmatrix_x4(uint32_t (&r)[4], const void* row) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(ptx::smem_u32(row)));
}
__device__ __forceinline__ void ldmatrix_x4_trans(uint32_t (&r)[4], const void* row) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(ptx::smem_u32(row)));
}
__device__ __forceinline__ void ldmatrix_x2_trans(uint32_t (&r)[2], const void* row) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x2.trans.shared.b16 {%0,%1}, [%2];"
                 : "=r"(r[0]), "=r"(r[1]) : "r"(ptx::smem_u32(row)));
}
// D += A (16x16, row) * B (16x8, col), bf16 inputs, fp32 accumulate.
__device__ __forceinline__ void mma_bf16_16816(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// The arithmetic runs on the tensor cores (mma.sync m16n8k16, bf16 x bf16 -> fp32):
//   scores : S[16 tokens x 8 heads] = K[16 x D] . Q^T[D x 8]  -- the query-head group of a KV head (up to 8
//            heads) is the N dimension; warp w owns tokens [16 w, 16 w + 16); keys and queries enter as the
//            bf16 numbers they are and the scale multiplies the fp32 sums;
//   softmax: one warp per head over the split's 128 scores (shared memory), fp32; the probabilities are
//            written as TWO bf16 numbers hi + lo (relative error 2^-17), so that the second product runs
//            on the tensor cores without giving up the fp32 probabilities of the reference;
//   values : O[8 heads x D] = P[8 x 128 tokens] . V[128 x D]  -- warp w owns D / 8 head-dim columns, the value
//            tile is read with transposing matrix loads, hi and lo are two MMAs into one accumulator.
// Measured against the CUDA-core form of the same kernel (one token per lane, FMAs against the queries in
// shared memory), which spent two thirds of its instructions on converts and shared-memory reads.
template <int kD, int kG>
__global__ void __launch_bounds__(kAttnThreads) attention_decode_split_kernel(const AttentionParams p) {
    constexpr int kRow = kD + kAttnRowPad;   // elements; the 16 bytes of padding keep matrix loads conflict-free
    constexpr int kSlices = kD / 16;         // k-steps of the score product
    constexpr int kColsPerWarp = kD / 8;     // head-dim columns a warp owns in the value product (16 or 8)
    constexpr int kNTiles = kColsPerWarp / 8;
    constexpr int kProbRow = kAttnSplitTokens + 8;
    extern __shared__ __align__(16) uint16_t tiles[];
    uint16_t* key_tile = tiles;                                // [128][kRow]
    uint16_t* value_tile = tiles + kAttnSplitTokens * kRow;    // [128][kRow]
    __shared__ __align__(16) uint16_t prob_hi[8][kProbRow], prob_lo[8][kProbRow];
    __shared__ float warp_max[8][8], warp_sum[8][8];           // [warp][head]

    const int split = blockIdx.x;
    const int bh = blockIdx.y;                     // b * Hkv + h
    const int b = bh / p.kv_heads, h = bh - b * p.kv_heads;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int g = lane >> 2, t = lane & 3;         // fragment coordinates
    ptx::griddep_launch_dependents();
    ptx::griddep_wait();                           // q and the newest cache row are the preceding kernels' output
    const int n = p.lengths ? p.lengths[b] : p.tokens;
    const size_t cache_row0 = ((size_t)bh * p.capacity) * kD;
    const int split_first = split * kAttnSplitTokens;
    const int rows = min(kAttnSplitTokens, n - split_first);  // tokens of this split in use (<= 0: none)
    // A split past the sequence's end has nothing to do and the merge never reads its partial (callers
    // pass whole caches with the lengths on the device, so most splits of a short sequence are such).
    if (rows <= 0 && p.splits > 1) return;

    // Both tiles are requested at once, 16 bytes per copy: every byte this CTA will read is in flight
    // before any arithmetic starts.  Two groups, so the score phase can begin when the keys are in.
    constexpr int kChunks = kD / 8;
    for (int c = threadIdx.x; c < rows * kChunks; c += kAttnThreads) {
        const int row = c / kChunks, chunk = c - row * kChunks;
        ptx::cp_async_16(key_tile + row * kRow + chunk * 8, p.k + cache_row0 + (size_t)(split_first + row) * kD + chunk * 8);
    }
    ptx::cp_async_commit();
    for (int c = threadIdx.x; c < rows * kChunks; c += kAttnThreads) {
        const int row = c / kChunks, chunk = c - row * kChunks;
        ptx::cp_async_16(value_tile + row * kRow + chunk * 8, p.v + cache_row0 + (size_t)(split_first + row) * kD + chunk * 8);
    }
    ptx::cp_async_commit();
    // Rows past the sequence's end enter the value product with probability zero; their bytes must
    // still be numbers (0 x NaN is NaN).  Key rows past the end only produce scores that are masked.
    const int first_unused = max(rows, 0);
    for (int c = threadIdx.x; c < (kAttnSplitTokens - first_unused) * kChunks; c += kAttnThreads) {
        const int row = first_unused + c / kChunks, chunk = c % kChunks;
        *reinterpret_cast<uint4*>(value_tile + row * kRow + chunk * 8) = make_uint4(0u, 0u, 0u, 0u);
        *reinterpret_cast<uint4*>(key_tile + row * kRow + chunk * 8) = make_uint4(0u, 0u, 0u, 0u);
    }

    // Query fragments (the B operand of the score product): head g, dims 16 s + 2 t (+1) and + 8.
    uint32_t qf[kSlices][2];
    {
        const uint16_t* qrow = p.q + ((size_t)b * p.q_heads + (size_t)h * kG + min(g, kG - 1)) * kD;
#pragma unroll
        for (int s = 0; s < kSlices; ++s) {
            uint32_t lo, hi;
            asm volatile("ld.global.u32 %0, [%1];" : "=r"(lo) : "l"(qrow + 16 * s + 2 * t));
            asm volatile("ld.global.u32 %0, [%1];" : "=r"(hi) : "l"(qrow + 16 * s + 2 * t + 8));
            qf[s][0] = g < kG ? lo : 0u;
            qf[s][1] = g < kG ? hi : 0u;
        }
    }
    ptx::cp_async_wait_group<1>();
    __syncthreads();

    // ---------------------------------------------------------------- scores: 16 tokens per warp
    // c0, c1: token 16 w + g, heads 2 t and 2 t + 1; c2, c3: token 16 w + g + 8.  The scores stay in
    // these registers through the softmax; only the per-warp maxima and sums meet in shared memory.
    float c[4] = {0.0f, 0.0f, 0.0f, 0.0f};
    {
        const uint16_t* a_row = key_tile + (16 * warp + (lane & 15)) * kRow + 8 * (lane >> 4);
#pragma unroll
        for (int s = 0; s < kSlices; ++s) {
            uint32_t a[4];
            ldmatrix_x4(a, a_row + 16 * s);
            mma_bf16_16816(c, a, qf[s][0], qf[s][1]);
        }
    }
    const int token0 = 16 * warp + g, token1 = token0 + 8;
    c[0] = token0 < rows ? c[0] * p.scale : -INFINITY;
    c[1] = token0 < rows ? c[1] * p.scale : -INFINITY;
    c[2] = token1 < rows ? c[2] * p.scale : -INFINITY;
    c[3] = token1 < rows ? c[3] * p.scale : -INFINITY;
    {
        float even = fmaxf(c[0], c[2]), odd = fmaxf(c[1], c[3]);   // heads 2 t and 2 t + 1 over this lane's tokens
#pragma unroll
        for (int offset = 4; offset <= 16; offset <<= 1) {        // over g: the warp's 16 tokens
            even = fmaxf(even, __shfl_xor_sync(0xFFFFFFFFu, even, offset));
            odd = fmaxf(odd, __shfl_xor_sync(0xFFFFFFFFu, odd, offset));
        }
        if (g == 0) {
            warp_max[warp][2 * t] = even;
            warp_max[warp][2 * t + 1] = odd;
        }
    }
    __syncthreads();
    // ---------------------------------------------------------------- softmax over the split's 128 tokens
    {
        float m_even = warp_max[0][2 * t], m_odd = warp_max[0][2 * t + 1];
#pragma unroll
        for (int w = 1; w < 8; ++w) {
            m_even = fmaxf(m_even, warp_max[w][2 * t]);
            m_odd = fmaxf(m_odd, warp_max[w][2 * t + 1]);
        }
        // Masked tokens: exp(-inf - m) = 0; a split with no token at all has m = -inf and contributes 0.
        const float e0 = m_even == -INFINITY ? 0.0f : __expf(c[0] - m_even);
        const float e1 = m_odd == -INFINITY ? 0.0f : __expf(c[1] - m_odd);
        const float e2 = m_even == -INFINITY ? 0.0f : __expf(c[2] - m_even);
        const float e3 = m_odd == -INFINITY ? 0.0f : __expf(c[3] - m_odd);
        float even = e0 + e2, odd = e1 + e3;
#pragma unroll
        for (int offset = 4; offset <= 16; offset <<= 1) {
            even += __shfl_xor_sync(0xFFFFFFFFu, even, offset);
            odd += __shfl_xor_sync(0xFFFFFFFFu, odd, offset);
        }
        if (g == 0) {
            warp_sum[warp][2 * t] = even;
            warp_sum[warp][2 * t + 1] = odd;
        }
        // The probabilities as hi + lo (two bf16 numbers each), [head][token]; heads past the group get
        // zeros (their queries were zero, so e = exp(0 - 0) = 1 must not reach the padded rows).
        const float e[4] = {e0, e1, e2, e3};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int head = 2 * t + (i & 1), token = i < 2 ? token0 : token1;
            const float value = head < kG ? e[i] : 0.0f;
            const uint16_t hi = f32_to_bf16_bits(value);
            prob_hi[head][token] = hi;
            prob_lo[head][token] = f32_to_bf16_bits(value - bf16_bits_to_f32(hi));
        }
    }
    ptx::cp_async_wait_group<0>();
    __syncthreads();  // values have landed and every probability is written
    // ---------------------------------------------------------------- values: D / 8 columns per warp
    float acc[kNTiles][4];
#pragma unroll
    for (int nt = 0; nt < kNTiles; ++nt)
#pragma unroll
        for (int i = 0; i < 4; ++i) acc[nt][i] = 0.0f;
    const int dim0 = warp * kColsPerWarp;
#pragma unroll
    for (int ks = 0; ks < kAttnSplitTokens / 16; ++ks) {
        if (16 * ks >= rows) break;  // whole k-steps past the end contribute nothing
        // A operand: P[head g][tokens 16 ks + 2 t (+1)] and + 8; rows 8..15 of the 16-row tile are zero.
        uint32_t a_hi[4], a_lo[4];
        a_hi[0] = *reinterpret_cast<const uint32_t*>(&prob_hi[g][16 * ks + 2 * t]);
        a_hi[2] = *reinterpret_cast<const uint32_t*>(&prob_hi[g][16 * ks + 2 * t + 8]);
        a_lo[0] = *reinterpret_cast<const uint32_t*>(&prob_lo[g][16 * ks + 2 * t]);
        a_lo[2] = *reinterpret_cast<const uint32_t*>(&prob_lo[g][16 * ks + 2 * t + 8]);
        a_hi[1] = a_hi[3] = a_lo[1] = a_lo[3] = 0u;
        if constexpr (kNTiles == 2) {
            uint32_t bfrag[4];
            ldmatrix_x4_trans(bfrag, value_tile + (16 * ks + (lane & 7) + ((lane >> 3) & 1) * 8) * kRow + dim0 + 8 * (lane >> 4));
            mma_bf16_16816(acc[0], a_hi, bfrag[0], bfrag[1]);
            mma_bf16_16816(acc[0], a_lo, bfrag[0], bfrag[1]);
            mma_bf16_16816(acc[1], a_hi, bfrag[2], bfrag[3]);
            mma_bf16_16816(acc[1], a_lo, bfrag[2], bfrag[3]);
        } else {
            uint32_t bfrag[2];
            ldmatrix_x2_trans(bfrag, value_tile + (16 * ks + (lane & 7) + ((lane >> 3) & 1) * 8) * kRow + dim0);
            mma_bf16_16816(acc[0], a_hi, bfrag[0], bfrag[1]);
            mma_bf16_16816(acc[0], a_lo, bfrag[0], bfrag[1]);
        }
    }
    // acc[nt][0], [1]: head g, dims dim0 + 8 nt + 2 t (+1); [2], [3] belong to the padded heads.
    if (g < kG) {
        float m = warp_max[0][g], total = warp_sum[0][g];
#pragma unroll
        for (int w = 1; w < 8; ++w) {   // the eight warps' sums in warp order
            m = fmaxf(m, warp_max[w][g]);
            total += warp_sum[w][g];
        }
#pragma unroll
        for (int nt = 0; nt < kNTiles; ++nt) {
            const int d = dim0 + 8 * nt + 2 * t;
            if (p.splits == 1) {
                const size_t at = ((size_t)b * p.q_heads + (size_t)h * kG + g) * kD + d;
                const uint32_t pair = pack_bf16x2(acc[nt][0] / total, acc[nt][1] / total);
                *reinterpret_cast<uint32_t*>(p.out + at) = pair;
            } else {
                float* row = p.partial + (((size_t)bh * p.splits + split) * kG + g) * (kD + 2);
                row[d] = acc[nt][0];
                row[d + 1] = acc[nt][1];
                if (d == 0) {
                    row[kD] = m;
                    row[kD + 1] = total;
                }
            }
        }
    }
}

// Merges the splits of one (sequence, query head) in split order.  Bound by latency: a thread has the partials of
// sixteen splits in flight, requested before it knows the maximum, and a lane of each warp has the weight of one
// split (with two loads at a time and the splits in series: one sequence of 8192 tokens, eight KV heads of four query
// heads, 19.1 us for both kernels, now 14.3; sixteen of 2048, two of six, 13.4 and 12.5).
template <int kD>
__global__ void __launch_bounds__(kD) attention_decode_merge_kernel(const AttentionParams p, int group) {
    constexpr int kAhead = 16;
    const int bq = blockIdx.x;                      // b * Hq + query head
    const int b = bq / p.q_heads, qh = bq - b * p.q_heads;
    const int h = qh / group, g = qh - h * group;
    const int d = threadIdx.x, lane = threadIdx.x & 31;
    ptx::griddep_launch_dependents();
    ptx::griddep_wait();
    const int n = p.lengths ? p.lengths[b] : p.tokens;
    const int used = min(p.splits, (n + kAttnSplitTokens - 1) / kAttnSplitTokens);
    const float* base = p.partial + (((size_t)(b * p.kv_heads + h) * p.splits) * group + g) * (kD + 2);
    const size_t stride = (size_t)group * (kD + 2);
    float ahead[kAhead];
#pragma unroll
    for (int i = 0; i < kAhead; ++i) ahead[i] = i < used ? base[i * stride + d] : 0.0f;
    const float first_max = lane < used ? base[lane * stride + kD] : -INFINITY;  // split `lane`
    const float first_sum = lane < used ? base[lane * stride + kD + 1] : 0.0f;
    float m = first_max;
    for (int s = 32 + lane; s < used; s += 32) m = fmaxf(m, base[s * stride + kD]);
#pragma unroll
    for (int offset = 16; offset >= 1; offset >>= 1) m = fmaxf(m, __shfl_xor_sync(0xFFFFFFFFu, m, offset));
    float total = 0.0f, value = 0.0f;
    for (int s0 = 0; s0 < used; s0 += 32) {
        const int s = s0 + lane;
        const float split_max = s0 == 0 ? first_max : s < used ? base[s * stride + kD] : -INFINITY;
        const float split_sum = s0 == 0 ? first_sum : s < used ? base[s * stride + kD + 1] : 0.0f;
        const float factor = __expf(split_max - m);
#pragma unroll
        for (int part = 0; part < 32; part += kAhead) {
            if (s0 + part >= used) break;
            float current[kAhead];
#pragma unroll
            for (int i = 0; i < kAhead; ++i) {
                const int next = s0 + part + kAhead + i;
                current[i] = ahead[i];
                if (next < used) ahead[i] = base[next * stride + d];
            }
#pragma unroll
            for (int i = 0; i < kAhead; ++i) {
                const float f = __shfl_sync(0xFFFFFFFFu, factor, part + i), t = __shfl_sync(0xFFFFFFFFu, split_sum, part + i);
                if (s0 + part + i < used) {
                    total = fmaf(t, f, total);
                    value = fmaf(current[i], f, value);
                }
            }
        }
    }
    p.out[(size_t)bq * kD + d] = f32_to_bf16_bits(value / total);
}

inline int attention_splits(int tokens) { return tokens <= 0 ? 1 : (tokens + kAttnSplitTokens - 1) / kAttnSplitTokens; }

inline size_t attention_workspace_bytes(int batch, int q_heads, int tokens, int head_dim) {
    const int splits = attention_splits(tokens);
    if (splits <= 1) return 0;
    return (size_t)batch * q_heads * splits * (head_dim + 2) * sizeof(float);
}

template <int kD, int kG>
inline int launch_attention_instance(const AttentionParams& params, int batch, cudaStream_t stream) {
    static bool configured[64] = {};
    int device = 0;
    cudaGetDevice(&device);
    if (device >= 64 || !configured[device]) {
        if (cudaFuncSetAttribute(attention_decode_split_kernel<kD, kG>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 attention_smem_bytes<kD>()) != cudaSuccess)
            return MT_ERR_LAUNCH;
        if (device < 64) configured[device] = true;
    }
    cudaLaunchConfig_t config = {};
    config.gridDim = dim3(params.splits, batch * params.kv_heads, 1);
    config.blockDim = dim3(kAttnThreads, 1, 1);
    config.dynamicSmemBytes = attention_smem_bytes<kD>();
    config.stream = stream;
    cudaLaunchAttribute attrs[1];
    attrs[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attrs[0].val.programmaticStreamSerializationAllowed = 1;
    config.attrs = attrs;
    config.numAttrs = 1;
    if (cudaLaunchKernelEx(&config, attention_decode_split_kernel<kD, kG>, params) != cudaSuccess) return MT_ERR_LAUNCH;
    if (params.splits > 1) {
        config.gridDim = dim3(batch * params.q_heads, 1, 1);
        config.blockDim = dim3(kD, 1, 1);
        config.dynamicSmemBytes = 0;
        if (cudaLaunchKernelEx(&config, attention_decode_merge_kernel<kD>, params, kG) != cudaSuccess)
            return MT_ERR_LAUNCH;
    }
    return MT_OK;
}

template <int kD>
inline int launch_attention_dim(const AttentionParams& params, int batch, int group, cudaStream_t stream) {
    switch (group) {
        case 1: return launch_attention_instance<kD, 1>(params, batch, stream);
        case 2: return launch_attention_instance<kD, 2>(params, batch, stream);
        case 3: return launch_attention_instance<kD, 3>(params, batch, stream);
        case 4: return launch_attention_instance<kD, 4>(params, batch, stream);
        case 5: return launch_attention_instance<kD, 5>(params, batch, stream);
        case 6: return launch_attention_instance<kD, 6>(params, batch, stream);
        case 7: return launch_attention_instance<kD, 7>(params, batch, stream);
        case 8: return launch_attention_instance<kD, 8>(params, batch, stream);
        default: return MT_ERR_SHAPE;
    }
}

// ---------------------------------------------------------------------------------------------
// Rotary embedding (half-split pairs (i, i + D/2), angle = position * theta^(-2i/D)) of the new
// query and key rows, and the append of the rotated key and of the value at `position` of each
// sequence's cache.  One CTA per sequence, a thread per pair of a head: the sequence's angles are computed once, and the
// CTA can advance the position itself, since no other one reads it.  Bound by latency: the rows are requested
// before the angles are known.  (A CTA per head, each with its own angles, and the framework's increment behind it, which
// also kept the next kernel's launch from overlapping, took 4.0 + 2.8 us.)
struct RopeAppendParams {
    const uint16_t* q;        // [B, Hq, D], consecutive sequences `row_stride` elements apart
    const uint16_t* k;        // [B, Hkv, D], same stride
    const uint16_t* v;        // [B, Hkv, D], same stride
    int* positions;           // [B]
    uint16_t* q_out;          // [B, Hq, D]
    uint16_t* k_cache;        // [B, Hkv, capacity, D]
    uint16_t* v_cache;
    int q_heads, kv_heads, capacity, head_dim;
    bool advance;             // add one to the positions
    long long row_stride;     // elements between sequences in q, k and v (one fused q|k|v row, or dense)
    float log2_theta;
};

constexpr int kRopeThreads = 1024;

__global__ void __launch_bounds__(kRopeThreads) rope_kv_append_kernel(const RopeAppendParams p) {
    extern __shared__ float rope_angles[];  // cosines, then sines
    const int b = blockIdx.x;
    const int dim = p.head_dim, half = dim >> 1;
    const int pairs = (p.q_heads + 2 * p.kv_heads) * half;
    ptx::griddep_launch_dependents();
    ptx::griddep_wait();
    auto row = [&](int slot) {
        const uint16_t* from = slot < p.q_heads ? p.q + (size_t)slot * dim
                             : slot < p.q_heads + p.kv_heads ? p.k + (size_t)(slot - p.q_heads) * dim
                                                             : p.v + (size_t)(slot - p.q_heads - p.kv_heads) * dim;
        return from + (size_t)b * p.row_stride;
    };
    int at = threadIdx.x, slot = at / half, i = at - slot * half;
    uint16_t first_bits = 0, second_bits = 0;
    if (at < pairs) {
        first_bits = ptx::ld_global_dependent_u16(row(slot) + i);
        second_bits = ptx::ld_global_dependent_u16(row(slot) + i + half);
    }
    const int position = p.positions[b];
    for (int pair = threadIdx.x; pair < half; pair += blockDim.x) {
        // theta^(-2i/D) = 2^(-(2i/D) log2 theta); sincosf on position * that, in fp32.
        const float inverse = exp2f(-(2.0f * (float)pair / (float)dim) * p.log2_theta);
        sincosf((float)position * inverse, &rope_angles[half + pair], &rope_angles[pair]);
    }
    __syncthreads();
    if (p.advance && threadIdx.x == 0) p.positions[b] = position + 1;
    while (at < pairs) {
        const int h = slot < p.q_heads ? slot : (slot - p.q_heads) % p.kv_heads;
        uint16_t* cache = slot < p.q_heads + p.kv_heads ? p.k_cache : p.v_cache;
        uint16_t* to = slot < p.q_heads ? p.q_out + ((size_t)b * p.q_heads + h) * dim
                                        : cache + (((size_t)b * p.kv_heads + h) * p.capacity + position) * dim;
        if (slot < p.q_heads + p.kv_heads) {
            const float c = rope_angles[i], s = rope_angles[half + i];
            const float first = bf16_bits_to_f32(first_bits), second = bf16_bits_to_f32(second_bits);
            to[i] = f32_to_bf16_bits(first * c - second * s);
            to[i + half] = f32_to_bf16_bits(second * c + first * s);
        } else {
            to[i] = first_bits;
            to[i + half] = second_bits;
        }
        at += blockDim.x;
        if (at < pairs) {
            slot = at / half;
            i = at - slot * half;
            first_bits = ptx::ld_global_dependent_u16(row(slot) + i);
            second_bits = ptx::ld_global_dependent_u16(row(slot) + i + half);
        }
    }
}

// The same for a prompt: `steps` new tokens of each sequence at rows `first`, `first + 1`, ... of its cache.  Every
// product, sum and difference is rounded by itself, the angle is position * inverse[pair], and cosf / sinf are those
// of the library: what the framework's op-by-op form computes, to the bit.  One CTA per token; its cosines and
// sines are computed once for all heads.  Bound by launch latency and bytes (512 tokens of 12 + 2 x 2 heads of 128:
// 4.4 us; as some 45 framework launches per layer, together with the head over all positions, 540 us per block).
struct RopePrefillParams {
    const uint16_t* q;        // [B, steps, Hq, D]
    const uint16_t* k;        // [B, steps, Hkv, D]
    const uint16_t* v;        // [B, steps, Hkv, D]
    const float* inverse;     // [D / 2]
    uint16_t* q_out;          // [B, steps, Hq, D]
    uint16_t* k_cache;        // [B, Hkv, capacity, D]
    uint16_t* v_cache;
    int* positions;           // [B] or null: advanced by `steps`
    int steps, first, q_heads, kv_heads, capacity, head_dim;
};

template <bool kVector>
__global__ void __launch_bounds__(256) rope_kv_prefill_kernel(const RopePrefillParams p) {
    extern __shared__ float rope_angles[];  // cosines, then sines
    const int b = blockIdx.x / p.steps, step = blockIdx.x - b * p.steps;
    const int dim = p.head_dim, half = dim >> 1;
    float *cosines = rope_angles, *sines = rope_angles + half;
    ptx::griddep_launch_dependents();
    ptx::griddep_wait();  // the table too may be the preceding kernel's output
    for (int i = threadIdx.x; i < half; i += blockDim.x) {
        const float angle = __fmul_rn((float)(p.first + step), p.inverse[i]);
        cosines[i] = cosf(angle);
        sines[i] = sinf(angle);
    }
    __syncthreads();
    if (step == 0 && threadIdx.x == 0 && p.positions) p.positions[b] += p.steps;
    constexpr int kWidth = kVector ? 8 : 1;   // pairs of a thread
    const int units = half / kWidth;          // threads of a head
    for (int at = threadIdx.x; at < (p.q_heads + 2 * p.kv_heads) * units; at += blockDim.x) {
        const int slot = at / units, i = (at - slot * units) * kWidth;
        const bool is_query = slot < p.q_heads;
        const int h = is_query ? slot : (slot - p.q_heads) % p.kv_heads;
        const bool is_value = slot >= p.q_heads + p.kv_heads;
        const uint16_t* from = is_query ? p.q + ((size_t)blockIdx.x * p.q_heads + h) * dim
                                        : (is_value ? p.v : p.k) + ((size_t)blockIdx.x * p.kv_heads + h) * dim;
        uint16_t* to = is_query ? p.q_out + ((size_t)blockIdx.x * p.q_heads + h) * dim
                                : (is_value ? p.v_cache : p.k_cache) + (((size_t)b * p.kv_heads + h) * p.capacity + p.first + step) * dim;
        auto rotate = [&](float first, float second, int pair, float& low, float& high) {
            const float c = cosines[pair], s = sines[pair];
            low = __fsub_rn(__fmul_rn(first, c), __fmul_rn(second, s));
            high = __fadd_rn(__fmul_rn(second, c), __fmul_rn(first, s));
        };
        if constexpr (kVector) {
            const uint4 a = ptx::ld_global_dependent_u4(from + i), z = ptx::ld_global_dependent_u4(from + i + half);
            uint4 low4 = a, high4 = z;
            if (!is_value) {
                const uint32_t first[4] = {a.x, a.y, a.z, a.w}, second[4] = {z.x, z.y, z.z, z.w};
                uint32_t low[4], high[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    float l0, h0, l1, h1;
                    rotate(bf16_lo(first[j]), bf16_lo(second[j]), i + 2 * j, l0, h0);
                    rotate(bf16_hi(first[j]), bf16_hi(second[j]), i + 2 * j + 1, l1, h1);
                    low[j] = pack_bf16x2(l0, l1);
                    high[j] = pack_bf16x2(h0, h1);
                }
                low4 = make_uint4(low[0], low[1], low[2], low[3]);
                high4 = make_uint4(high[0], high[1], high[2], high[3]);
            }
            *reinterpret_cast<uint4*>(to + i) = low4;
            *reinterpret_cast<uint4*>(to + i + half) = high4;
        } else {
            const uint16_t a = ptx::ld_global_dependent_u16(from + i), z = ptx::ld_global_dependent_u16(from + i + half);
            float low, high;
            rotate(bf16_bits_to_f32(a), bf16_bits_to_f32(z), i, low, high);
            to[i] = is_value ? a : f32_to_bf16_bits(low);
            to[i + half] = is_value ? z : f32_to_bf16_bits(high);
        }
    }
}

// ---------------------------------------------------------------------------------------------
// The end of a greedy decode step: a row of bf16 logits as fp32, and the index of its largest value (the first one
// of equals, a NaN before any number) as the next step's token.  A cluster of eight CTAs shares a row: every CTA
// converts its part and leaves its candidate with CTA 0.  Bound by latency (16 rows of 32768 as
// three framework launches for the conversion, the maximum's index and a copy: 5.8 + 14.8 + 2.5 us; with it and the
// rotary kernel above a decode step of sixteen sequences through four blocks takes 243 us, 259 before).
struct GreedyParams {
    const uint16_t* logits;   // [rows, vocabulary]
    float* out;               // [rows, vocabulary]
    long long* tokens;        // [rows]
    int vocabulary;
};

constexpr int kGreedyThreads = 256, kGreedyCluster = 8;
// Beyond the limits a loop's next index or the grid would not fit an int.
static_assert(MT_GREEDY_MAX_VOCABULARY <= 0x7FFFFFFF - kGreedyThreads * kGreedyCluster * 8 && MT_GREEDY_MAX_ROWS <= 0x7FFFFFFF / kGreedyCluster, "int overflow");

struct GreedyCandidate {
    float value;
    int index;
};

__device__ __forceinline__ GreedyCandidate greedy_better(GreedyCandidate a, GreedyCandidate b) {
    const bool a_nan = a.value != a.value, b_nan = b.value != b.value;
    const bool same = a_nan ? b_nan : a.value == b.value;
    const bool take_a = same ? a.index < b.index : a_nan || (!b_nan && a.value > b.value);
    return take_a ? a : b;
}

template <bool kVector>
__global__ void __launch_bounds__(kGreedyThreads) greedy_token_kernel(const GreedyParams p) {
    __shared__ GreedyCandidate found[kGreedyThreads / 32];
    __shared__ float cluster_values[kGreedyCluster], cluster_indexes[kGreedyCluster];
    const int rank = ptx::cluster_ctarank(), row = blockIdx.x / kGreedyCluster;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    ptx::cluster_arrive();  // every CTA of the cluster has started: its shared memory may be written below
    ptx::griddep_launch_dependents();
    ptx::griddep_wait();
    const uint16_t* from = p.logits + (size_t)row * p.vocabulary;
    float* to = p.out + (size_t)row * p.vocabulary;
    GreedyCandidate best = {-INFINITY, 0x7FFFFFFF};
    if constexpr (kVector) {
        for (int i = (rank * kGreedyThreads + threadIdx.x) * 8; i < p.vocabulary; i += kGreedyCluster * kGreedyThreads * 8) {
            const uint4 v = ptx::ld_global_dependent_u4(from + i);
            const uint32_t words[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const float low = bf16_lo(words[j]), high = bf16_hi(words[j]);
                best = greedy_better(best, {low, i + 2 * j});
                best = greedy_better(best, {high, i + 2 * j + 1});
            }
            *reinterpret_cast<float4*>(to + i) = make_float4(bf16_lo(v.x), bf16_hi(v.x), bf16_lo(v.y), bf16_hi(v.y));
            *reinterpret_cast<float4*>(to + i + 4) = make_float4(bf16_lo(v.z), bf16_hi(v.z), bf16_lo(v.w), bf16_hi(v.w));
        }
    } else {
        for (int i = rank * kGreedyThreads + threadIdx.x; i < p.vocabulary; i += kGreedyCluster * kGreedyThreads) {
            const float v = bf16_bits_to_f32(ptx::ld_global_dependent_u16(from + i));
            best = greedy_better(best, {v, i});
            to[i] = v;
        }
    }
    auto across_lanes = [&](int first_offset) {
        for (int offset = first_offset; offset >= 1; offset >>= 1) {
            const GreedyCandidate other = {__shfl_xor_sync(0xFFFFFFFFu, best.value, offset), __shfl_xor_sync(0xFFFFFFFFu, best.index, offset)};
            best = greedy_better(best, other);
        }
    };
    across_lanes(16);
    if (lane == 0) found[warp] = best;
    __syncthreads();
    ptx::cluster_wait();
    if (warp == 0) {
        if (lane < kGreedyThreads / 32) best = found[lane];
        across_lanes(kGreedyThreads / 64);
        if (lane == 0) {  // the index travels as the float of its bits
            ptx::st_cluster_f32(ptx::map_to_cta(ptx::smem_u32(&cluster_values[rank]), 0), best.value);
            ptx::st_cluster_f32(ptx::map_to_cta(ptx::smem_u32(&cluster_indexes[rank]), 0), __int_as_float(best.index));
        }
        __syncwarp();
    }
    ptx::cluster_arrive();
    ptx::cluster_wait();
    if (rank == 0 && warp == 0) {
        if (lane < kGreedyCluster) best = {cluster_values[lane], __float_as_int(cluster_indexes[lane])};
        across_lanes(kGreedyCluster / 2);
        if (lane == 0) p.tokens[row] = best.index;
    }
}

}  // namespace mt
