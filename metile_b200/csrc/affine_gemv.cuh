// INT4 affine dequant-GEMV on the CUDA cores, for 1..8 activation rows served from ONE read of
// the packed weights.
//
// Computes what the reference's kernels/affine_qmv.py:4-54 computes (word / element / group
// indexing, w = scale*q + bias, fp32 accumulation, one rounding at the store) with the residual
// epilogue of :124-131 and the SwiGLU epilogue of :204-208.  Unlike the reference's kernel, which
// re-reads the weights once per activation row (flattened output index, :22-24), every row of the
// batch shares the same weight registers here.
//
// Mapping: half a warp (16 lanes) owns one output row; lane l reads the 128-bit word group
// j = l + 16*t of that row (32 nibbles = half a scale group), t = 0, 1, ...  A warp pass covers
// 2*kRows output rows.  When N is small the K range of a row is cut into `ksplit` contiguous
// parts handled by different warps of the CTA (more bytes in flight); the parts are summed
// through shared memory in part order.  ksplit is a function of (N, K) only.
//
// Arithmetic.  The kernel is bound by instruction issue, not by HBM (the logic pipe runs at half
// the FMA pipe's rate), so a nibble costs two instructions: one byte-permute puts it into the
// mantissa of 128.0f, giving the float 128+q exactly, and one FMA multiplies it with the
// activation.  Per 32-nibble slot:  dot = sum_e (128+q_e) * x_e  in ascending e, then
//     acc = fma(scale, dot, fma(bias - 128*scale, xsum, acc)),   xsum = ((x_0 + x_1) + ...) + x_31,
// which equals scale*sum(q*x) + bias*sum(x) up to fp32 rounding.  Weights are never rounded.
// With one activation row the activations are converted to fp32 once per CTA and kept in shared
// memory in the order the lanes read them (16-byte chunks of consecutive lanes adjacent: no bank
// conflicts), together with the per-slot sums; with more rows they are converted on the fly.
// The order of every fp32 operation for one (row, output) pair depends on K only -- not on the
// number of rows, the grid, N or where the activations are staged -- so results are bit-identical
// for a row run alone or inside a batch of up to 8.
#pragma once

#include <algorithm>

#include "common.cuh"
#include "ptx.cuh"

namespace mt {

__device__ __forceinline__ uint4 ldg_stream_u4(const uint4* p) {
    uint4 v;
    asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];"
                 : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
                 : "l"(p));
    return v;
}

struct GemvWeights {
    const uint32_t* w;
    const uint16_t* scales;
    const uint16_t* biases;
};

enum GemvStage : int {
    kStageNone = 0,  // activations read from global memory
    kStageBf16 = 1,  // copied to shared memory as they are
    kStageF32 = 2,   // one row: converted to fp32, lane-interleaved, plus per-slot sums
};

// Shared-memory bytes of the kStageF32 layout: ceil(K/512) steps x 8 chunks x 16 lanes x 16 B, then
// one fp32 sum per 32-column slot.
inline int gemv_f32_stage_bytes(int K) {
    const int steps = ((K >> 5) + 15) >> 4;
    return steps * 8 * 16 * 16 + (K >> 5) * 4;
}

// kM rows of activations; kRows output rows per half-warp per pass; kDual = gate|up with SwiGLU.
//
// The (pass, slot) iteration space is flattened and software-pipelined: the packed words, scale and
// bias of iteration i+1 are requested before iteration i is computed.  With programmatic dependent
// launch the first request goes out before the kernel waits for its predecessor (nobody writes
// weights); the activations -- the predecessor's output -- are read only after that wait, with
// coherent loads.
template <int kM, int kRows, bool kDual, int kStage>
__global__ void __launch_bounds__(256)
affine_gemv_kernel(const uint16_t* x, GemvWeights first, GemvWeights second, const uint16_t* residual,
                   uint16_t* __restrict__ out, int K, int N, int ksplit) {
    static_assert(kStage != kStageF32 || kM == 1, "the fp32 stage holds one activation row");
    constexpr int kStreams = kDual ? 2 : 1;
    constexpr int kWarps = 8;
    extern __shared__ uint4 x_shared[];  // kStageBf16: [kM][K/8] vectors of 8 bf16; kStageF32: see above
    __shared__ float partial[kWarps][2][kStreams * kRows * kM];
    const int lane = threadIdx.x & 31;
    const int half = lane >> 4;
    const int l16 = lane & 15;
    const int warp = threadIdx.x >> 5;
    const int part = warp % ksplit;          // which K part this warp sums
    const int team = warp / ksplit;          // which row group of the CTA it belongs to
    const int teams_per_cta = kWarps / ksplit;
    const int slots_per_row = K >> 5;  // 128-bit word groups per weight row
    const int words_per_row = K >> 3;
    const int groups_per_row = K >> 6;
    const int rows_per_pass = 2 * kRows;
    const int slots_per_part = (slots_per_row + ksplit - 1) / ksplit;
    const int slot_begin = part * slots_per_part;
    const int slot_end = min(slot_begin + slots_per_part, slots_per_row);
    const int team_global = blockIdx.x * teams_per_cta + team;
    const int teams_total = gridDim.x * teams_per_cta;
    // A CTA's row blocks (rows_per_pass rows per team) are blockIdx.x, blockIdx.x + gridDim.x, ...: it
    // runs as many passes as it has blocks that start below N -- not the grid-wide maximum, which at
    // N = 8192 made most CTAs spend a second pass on clamped rows whose results nobody stores, in a
    // kernel bound by instruction issue.  Every warp of a CTA runs the same number of iterations (the
    // bounds depend on blockIdx only), so the __syncthreads below are reached by all of them.
    const int row_blocks = (N + teams_per_cta * rows_per_pass - 1) / (teams_per_cta * rows_per_pass);
    const int passes = (int)((unsigned int)(row_blocks - 1 - (int)blockIdx.x) / gridDim.x) + 1;  // the grid has at most row_blocks CTAs
    const int steps = (slots_per_part + 15) >> 4;  // slot iterations per pass (some lanes idle in the last)

    struct Weights {
        uint4 packed[kStreams][kRows];
        uint32_t scale[kStreams][kRows], bias[kStreams][kRows];
    };
    auto request = [&](int pass, int step, Weights& w) {
        const int slot = slot_begin + l16 + (step << 4);
        if (pass >= passes || slot >= slot_end) return;
        const int row_base = (pass * teams_total + team_global) * rows_per_pass;
#pragma unroll
        for (int s = 0; s < kStreams; ++s) {
            const GemvWeights& wt = s == 0 ? first : second;
#pragma unroll
            for (int r = 0; r < kRows; ++r) {
                const int n = min(row_base + half * kRows + r, N - 1);  // clamp loads; the store is guarded
                w.packed[s][r] = ldg_stream_u4(reinterpret_cast<const uint4*>(wt.w + (size_t)n * words_per_row) + slot);
                const size_t g = (size_t)n * groups_per_row + (slot >> 1);
                w.scale[s][r] = __ldg(wt.scales + g);
                w.bias[s][r] = __ldg(wt.biases + g);
            }
        }
    };

    ptx::griddep_launch_dependents();
    Weights next;
    request(0, 0, next);
    ptx::griddep_wait();  // activations and residual are the preceding kernel's output
    if constexpr (kStage == kStageBf16) {
        const int vectors = kM * (K >> 3);
        for (int v = threadIdx.x; v < vectors; v += blockDim.x) x_shared[v] = ptx::ld_global_dependent_u4(x + (size_t)v * 8);
        __syncthreads();
    }
    if constexpr (kStage == kStageF32) {
        float4* xq = reinterpret_cast<float4*>(x_shared);
        const int steps_all = (slots_per_row + 15) >> 4;
        float* slot_sum = reinterpret_cast<float*>(xq + steps_all * 128);
        // Eight bf16 = chunks 2c and 2c+1 of their slot; chunk i of slot j lives at ((j/16)*8 + i)*16 + j%16.
        for (int v = threadIdx.x; v < (K >> 3); v += blockDim.x) {
            const uint4 raw = ptx::ld_global_dependent_u4(x + (size_t)v * 8);
            const int slot = v >> 2, chunk = (v & 3) << 1;
            float4* dst = xq + (((slot >> 4) << 3) + chunk) * 16 + (slot & 15);
            dst[0] = make_float4(bf16_lo(raw.x), bf16_hi(raw.x), bf16_lo(raw.y), bf16_hi(raw.y));
            dst[16] = make_float4(bf16_lo(raw.z), bf16_hi(raw.z), bf16_lo(raw.w), bf16_hi(raw.w));
        }
        __syncthreads();
        for (int slot = threadIdx.x; slot < slots_per_row; slot += blockDim.x) {
            const float4* src = xq + ((slot >> 4) << 3) * 16 + (slot & 15);
            float sum = 0.0f;
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const float4 c = src[i * 16];
                sum += c.x; sum += c.y; sum += c.z; sum += c.w;
            }
            slot_sum[slot] = sum;
        }
        __syncthreads();
    }

    float acc[kStreams][kRows][kM];
    int next_pass = 0, next_step = 0;
    for (int pass = 0; pass < passes; ++pass) {
        const int row_base = (pass * teams_total + team_global) * rows_per_pass;
#pragma unroll
        for (int s = 0; s < kStreams; ++s)
#pragma unroll
            for (int r = 0; r < kRows; ++r)
#pragma unroll
                for (int m = 0; m < kM; ++m) acc[s][r][m] = 0.0f;

        for (int step = 0; step < steps; ++step) {
            const int slot = slot_begin + l16 + (step << 4);
            const Weights cur = next;
            if (++next_step == steps) {
                next_step = 0;
                ++next_pass;
            }
            request(next_pass, next_step, next);
            if (slot >= slot_end) continue;

            float dot[kStreams][kRows][kM];
            float xsum[kM];
#pragma unroll
            for (int m = 0; m < kM; ++m) {
                xsum[m] = 0.0f;
#pragma unroll
                for (int s = 0; s < kStreams; ++s)
#pragma unroll
                    for (int r = 0; r < kRows; ++r) dot[s][r][m] = 0.0f;
            }
#pragma unroll
            for (int wi = 0; wi < 4; ++wi) {
                float xv[kM][8];
                if constexpr (kStage == kStageF32) {
                    const float4* src = reinterpret_cast<const float4*>(x_shared) + (((slot >> 4) << 3) + 2 * wi) * 16 + (slot & 15);
                    const float4 a = src[0], b = src[16];
                    xv[0][0] = a.x; xv[0][1] = a.y; xv[0][2] = a.z; xv[0][3] = a.w;
                    xv[0][4] = b.x; xv[0][5] = b.y; xv[0][6] = b.z; xv[0][7] = b.w;
                } else {
#pragma unroll
                    for (int m = 0; m < kM; ++m) {
                        uint4 raw;
                        if constexpr (kStage == kStageBf16) raw = x_shared[m * (K >> 3) + slot * 4 + wi];
                        else raw = ptx::ld_global_dependent_u4(x + (size_t)m * K + (size_t)slot * 32 + wi * 8);
                        xv[m][0] = bf16_lo(raw.x); xv[m][1] = bf16_hi(raw.x);
                        xv[m][2] = bf16_lo(raw.y); xv[m][3] = bf16_hi(raw.y);
                        xv[m][4] = bf16_lo(raw.z); xv[m][5] = bf16_hi(raw.z);
                        xv[m][6] = bf16_lo(raw.w); xv[m][7] = bf16_hi(raw.w);
#pragma unroll
                        for (int e = 0; e < 8; ++e) xsum[m] += xv[m][e];
                    }
                }
#pragma unroll
                for (int s = 0; s < kStreams; ++s)
#pragma unroll
                    for (int r = 0; r < kRows; ++r) {
                        const uint32_t word = wi == 0 ? cur.packed[s][r].x
                                            : wi == 1 ? cur.packed[s][r].y
                                            : wi == 2 ? cur.packed[s][r].z
                                                      : cur.packed[s][r].w;
                        float q[8];
                        unpack_word_f32_offset128(word, q);
#pragma unroll
                        for (int m = 0; m < kM; ++m)
#pragma unroll
                            for (int e = 0; e < 8; ++e) dot[s][r][m] = fmaf(q[e], xv[m][e], dot[s][r][m]);
                    }
            }
            if constexpr (kStage == kStageF32) {
                const float4* base = reinterpret_cast<const float4*>(x_shared);
                xsum[0] = reinterpret_cast<const float*>(base + ((slots_per_row + 15) >> 4) * 128)[slot];
            }
#pragma unroll
            for (int s = 0; s < kStreams; ++s)
#pragma unroll
                for (int r = 0; r < kRows; ++r) {
                    const float scale = bf16_bits_to_f32(cur.scale[s][r]), bias = bf16_bits_to_f32(cur.bias[s][r]);
                    const float shifted = fmaf(-128.0f, scale, bias);  // the weights were decoded as 128+q
#pragma unroll
                    for (int m = 0; m < kM; ++m)
                        acc[s][r][m] = fmaf(scale, dot[s][r][m], fmaf(shifted, xsum[m], acc[s][r][m]));
                }
        }

        // ---- end of a pass: 16-lane butterfly inside each half-warp, then the K parts in order
#pragma unroll
        for (int s = 0; s < kStreams; ++s)
#pragma unroll
            for (int r = 0; r < kRows; ++r)
#pragma unroll
                for (int m = 0; m < kM; ++m) {
                    float v = acc[s][r][m];
#pragma unroll
                    for (int offset = 8; offset >= 1; offset >>= 1) v += __shfl_xor_sync(0xFFFFFFFFu, v, offset);
                    acc[s][r][m] = v;
                }
        if (ksplit > 1) {
            if (l16 == 0) {
#pragma unroll
                for (int s = 0; s < kStreams; ++s)
#pragma unroll
                    for (int r = 0; r < kRows; ++r)
#pragma unroll
                        for (int m = 0; m < kM; ++m) partial[warp][half][(s * kRows + r) * kM + m] = acc[s][r][m];
            }
            __syncthreads();
            if (part == 0 && l16 == 0) {
#pragma unroll
                for (int s = 0; s < kStreams; ++s)
#pragma unroll
                    for (int r = 0; r < kRows; ++r)
#pragma unroll
                        for (int m = 0; m < kM; ++m) {
                            float v = acc[s][r][m];
                            for (int p = 1; p < ksplit; ++p) v += partial[warp + p][half][(s * kRows + r) * kM + m];
                            acc[s][r][m] = v;
                        }
            }
            __syncthreads();
        }
        if (part == 0 && l16 == 0) {
#pragma unroll
            for (int r = 0; r < kRows; ++r) {
                const int n = row_base + half * kRows + r;
                if (n < N) {
#pragma unroll
                    for (int m = 0; m < kM; ++m) {
                        float v;
                        if constexpr (kDual) v = swiglu_f32(acc[0][r][m], acc[kStreams - 1][r][m]);
                        else v = acc[0][r][m];
                        if (residual) v += bf16_bits_to_f32(ptx::ld_global_dependent_u16(residual + (size_t)m * N + n));
                        out[(size_t)m * N + n] = f32_to_bf16_bits(v);
                    }
                }
            }
        }
    }
}

// ---- one activation row, weights through per-warp rings --------------------------------------------
// The same sums in the same order as affine_gemv_kernel<1, ...>; what differs is how the operands get there.
// Weights requested into registers one iteration ahead cost 125 registers a thread, and a warp waits for all of an
// iteration's loads together.  Here every lane
// copies its own 16 bytes of packed words, and a warp the words that hold its scales and biases, into a ring of the
// warp's, two iterations ahead, by asynchronous copies (64 KB of words and up to 10 KB of tables in flight per SM, no registers, and no synchronisation
// beyond the warp's).  The fp32 activations and the slot sums are made by one thread per slot with one barrier; the
// lanes' totals of all rows are folded together (5 exchanges instead of 16); the warps' rows are dealt out SM by SM.
// Times in a replayed graph, with registers and with rings: 1536 -> 8960 6.8 and 4.7 us, 4096 -> 4096 7.6 and 5.0, 2048 ->
// 16384 10.3 and 7.1, 2048 -> 128256 42.2 and 37.6.  The largest are bound by the logic pipe: 44 instructions per 32
// weights for the unpack and 12 more beside it, at half rate, in a warp that issues 117.  Three CTAs of 80 registers
// per SM instead of two of 125: 38.5 us.
constexpr int kGemvRingSlots = 3;
constexpr int kGemvRingRows = 4;  // weight rows of a half-warp: four outputs, or two of gate and two of up
constexpr int kGemvTableWords = 5;  // nine groups of a row and step, wherever they start within a word
constexpr int kGemvRingBytes = 8 * kGemvRingSlots * kGemvRingRows * (32 * 16 + 2 * 2 * kGemvTableWords * 4);  // of a CTA of eight warps

template <bool kDual>
__global__ void __launch_bounds__(256, 2)
affine_gemv_ring_kernel(const uint16_t* x, GemvWeights first, GemvWeights second, const uint16_t* residual, uint16_t* out,
                        int K, int N, int ksplit) {
    constexpr int kStreams = kDual ? 2 : 1, kRows = kGemvRingRows / kStreams, kWarps = 8;
    constexpr int kTableSlot = kGemvRingRows * 4 * kGemvTableWords;  // words
    extern __shared__ uint4 gemv_smem[];
    __shared__ float partial[kWarps][2][kGemvRingRows];
    const int lane = threadIdx.x & 31, half = lane >> 4, l16 = lane & 15, warp = threadIdx.x >> 5;
    const int part = warp % ksplit, team = warp / ksplit, teams = kWarps / ksplit;
    const int slots_per_row = K >> 5, groups_per_row = K >> 6;
    const int slots_per_part = (slots_per_row + ksplit - 1) / ksplit;
    const int slot_begin = part * slots_per_part, slot_end = min(slot_begin + slots_per_part, slots_per_row);
    const int steps = (slots_per_part + 15) >> 4;
    const int tasks = (N + 2 * kRows - 1) / (2 * kRows);  // a task is the 2 kRows outputs of one warp pass
    const int stride = teams * gridDim.x;
    const int first_task = team * gridDim.x + blockIdx.x;

    // [slot][row][lane] 16 bytes, then [slot][row][scales, biases][half][kGemvTableWords] words.
    uint4* ring = gemv_smem + warp * (kGemvRingSlots * kGemvRingRows * 32) + lane;
    uint32_t* table_ring = reinterpret_cast<uint32_t*>(gemv_smem + kWarps * kGemvRingSlots * kGemvRingRows * 32) +
                           warp * (kGemvRingSlots * kTableSlot) + half * kGemvTableWords;
    float4* xq = reinterpret_cast<float4*>(gemv_smem) + kGemvRingBytes / 16;
    float* slot_sum = reinterpret_cast<float*>(xq + ((slots_per_row + 15) >> 4) * 128);

    // The first row of this half-warp in a task; the last task repeats some of its neighbour's rows.
    auto task_row = [&](int task) { return min(task * 2 * kRows + half * kRows, N - kRows); };
    // Byte offsets of the next packed words of each row, and of the first table word that this lane copies: lane 4 r + i of
    // a half-warp has word i of row r, for 4 bytes per lane would be sixteen times the bytes and as many accesses to
    // shared memory as all else together (131072 rows of 1024: 23.5 us).
    uint32_t word_at[kRows], table_at = 0;
    const int table_row = l16 >> 2, table_word = l16 & 3;
    const int group_begin = slot_begin >> 1, group_end = (slot_end + 1) >> 1;
    int table_left = 0;         // groups from the word's first one to the end of the part
    bool table_fifth = false;
    int copy_task = first_task, copy_step = 0;
    auto start_copies = [&] {
        const int n = task_row(copy_task);
#pragma unroll
        for (int r = 0; r < kRows; ++r) word_at[r] = (uint32_t)(n + r) * (uint32_t)(K >> 1) + (slot_begin + l16) * 16;
        const uint32_t entry = (uint32_t)(n + table_row % kRows) * groups_per_row + group_begin;
        table_at = ((entry >> 1) + table_word) * 4;
        table_left = group_end - group_begin + (int)(entry & 1u) - 2 * table_word;
        table_fifth = table_word == 0 && ((entry | slot_begin) & 1u);
    };
    start_copies();
    auto copy_next = [&](int ring_slot) {
        if (copy_task < tasks) {
            uint8_t* to = reinterpret_cast<uint8_t*>(ring) + ring_slot * (kGemvRingRows * 512);
            uint32_t* table_to = table_ring + ring_slot * kTableSlot + table_row * (4 * kGemvTableWords) + table_word;
            if (slot_begin + l16 + (copy_step << 4) < slot_end) {
#pragma unroll
                for (int r = 0; r < kGemvRingRows; ++r)
                    ptx::cp_async_16(to + r * 512, reinterpret_cast<const uint8_t*>((r < kRows ? first : second).w) + word_at[r % kRows]);
            }
            const GemvWeights& wt = kDual && table_row >= kRows ? second : first;
            const uint8_t* scales = reinterpret_cast<const uint8_t*>(wt.scales) + table_at;
            const uint8_t* biases = reinterpret_cast<const uint8_t*>(wt.biases) + table_at;
            // Of a word that holds one more group of the part, the rest may lie past the end of the array: it is read alone.
            auto copy_table_word = [&](int word, int left) {
                uint32_t* to = table_to + word;
                if (left > 1) {
                    ptx::cp_async_4(to, scales + 4 * word);
                    ptx::cp_async_4(to + 2 * kGemvTableWords, biases + 4 * word);
                } else if (left == 1) {
                    to[0] = *reinterpret_cast<const uint16_t*>(scales + 4 * word);
                    to[2 * kGemvTableWords] = *reinterpret_cast<const uint16_t*>(biases + 4 * word);
                }
            };
            copy_table_word(0, table_left);
            if (table_fifth) copy_table_word(4, table_left - 8);
        }
        ptx::cp_async_commit();
        if (++copy_step == steps) {
            copy_step = 0;
            copy_task += stride;
            start_copies();
        } else {
#pragma unroll
            for (int r = 0; r < kRows; ++r) word_at[r] += 256;
            table_at += 16;
            table_left -= 8;
        }
    };

    ptx::griddep_launch_dependents();
#pragma unroll
    for (int i = 0; i < kGemvRingSlots - 1; ++i) copy_next(i);
    ptx::griddep_wait();  // activations and residual are the preceding kernel's output
    for (int slot = threadIdx.x; slot < slots_per_row; slot += blockDim.x) {
        uint4 raw[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) raw[i] = ptx::ld_global_dependent_u4(x + (size_t)slot * 32 + i * 8);
        float4* dst = xq + (slot >> 4) * 128 + (slot & 15);  // chunk i of slot j lies at ((j / 16) * 8 + i) * 16 + j % 16
        float sum = 0.0f;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float4 a = make_float4(bf16_lo(raw[i].x), bf16_hi(raw[i].x), bf16_lo(raw[i].y), bf16_hi(raw[i].y));
            const float4 b = make_float4(bf16_lo(raw[i].z), bf16_hi(raw[i].z), bf16_lo(raw[i].w), bf16_hi(raw[i].w));
            dst[32 * i] = a;
            dst[32 * i + 16] = b;
            sum += a.x; sum += a.y; sum += a.z; sum += a.w;
            sum += b.x; sum += b.y; sum += b.z; sum += b.w;
        }
        slot_sum[slot] = sum;
    }
    __syncthreads();

    int ring_slot = 0;
    // Every warp of a CTA makes the same number of passes: the barriers below are reached by all of them.
    for (int task0 = blockIdx.x; task0 < tasks; task0 += stride) {
        const int task = task0 + team * gridDim.x;
        const int row = task_row(task);
        // Where this lane's scale lies among the table words of even and odd rows, the same in every step.
        const int offset = ((slot_begin + l16) >> 1) - group_begin;
        const uint32_t entry = (uint32_t)row * groups_per_row + group_begin;
        const uint32_t half_at[2] = {offset + (entry & 1u), offset + ((entry ^ groups_per_row) & 1u)};
        float acc[kGemvRingRows] = {};
        for (int step = 0; step < steps; ++step) {
            ptx::cp_async_wait_group<kGemvRingSlots - 2>();
            __syncwarp();
            copy_next(ring_slot == 0 ? kGemvRingSlots - 1 : ring_slot - 1);  // the slot that was read before this one
            const uint4* words = ring + ring_slot * (kGemvRingRows * 32);
            const uint16_t* tables = reinterpret_cast<const uint16_t*>(table_ring + ring_slot * kTableSlot);
            if (++ring_slot == kGemvRingSlots) ring_slot = 0;
            const int slot = slot_begin + l16 + (step << 4);
            if (task >= tasks || slot >= slot_end) continue;
            const float4* xs = xq + (slot >> 4) * 128 + (slot & 15);
            uint4 packed[kGemvRingRows];
            float dot[kGemvRingRows];
#pragma unroll
            for (int r = 0; r < kGemvRingRows; ++r) {
                packed[r] = words[r * 32];
                dot[r] = 0.0f;
            }
#pragma unroll
            for (int wi = 0; wi < 4; ++wi) {
                const float4 a = xs[32 * wi], b = xs[32 * wi + 16];
                const float xv[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
#pragma unroll
                for (int r = 0; r < kGemvRingRows; ++r) {
                    float q[8];
                    unpack_word_f32_offset128(wi == 0 ? packed[r].x : wi == 1 ? packed[r].y : wi == 2 ? packed[r].z : packed[r].w, q);
#pragma unroll
                    for (int e = 0; e < 8; ++e) dot[r] = fmaf(q[e], xv[e], dot[r]);
                }
            }
            const float xsum = slot_sum[slot];
#pragma unroll
            for (int r = 0; r < kGemvRingRows; ++r) {
                const float scale = bf16_bits_to_f32(tables[r * (8 * kGemvTableWords) + half_at[r % kRows & 1]]);
                const float bias = bf16_bits_to_f32(tables[r * (8 * kGemvTableWords) + 4 * kGemvTableWords + half_at[r % kRows & 1]]);
                acc[r] = fmaf(scale, dot[r], fmaf(fmaf(-128.0f, scale, bias), xsum, acc[r]));
            }
        }

        // The 16-lane butterfly of the four rows: after two halvings a lane has the sums of row l16 / 4.
        {
            const bool upper8 = l16 & 8, upper4 = l16 & 4;
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                const float keep = upper8 ? acc[i + 2] : acc[i], send = upper8 ? acc[i] : acc[i + 2];
                acc[i] = keep + __shfl_xor_sync(0xFFFFFFFFu, send, 8);
            }
            const float keep = upper4 ? acc[1] : acc[0], send = upper4 ? acc[0] : acc[1];
            acc[0] = keep + __shfl_xor_sync(0xFFFFFFFFu, send, 4);
            acc[0] += __shfl_xor_sync(0xFFFFFFFFu, acc[0], 2);
            acc[0] += __shfl_xor_sync(0xFFFFFFFFu, acc[0], 1);
        }
        float total = acc[0];
        if (ksplit > 1) {  // the K parts in order
            if ((l16 & 3) == 0) partial[warp][half][l16 >> 2] = total;
            __syncthreads();
            if (part == 0)
                for (int q = 1; q < ksplit; ++q) total += partial[warp + q][half][l16 >> 2];
            __syncthreads();
        }
        const float other = kDual ? __shfl_down_sync(0xFFFFFFFFu, total, 8) : 0.0f;  // up, whose rows are two further on
        const int n = row + (l16 >> 2);
        if (part == 0 && task < tasks && (l16 & 3) == 0 && (l16 >> 2) < kRows && n >= task * 2 * kRows + half * kRows) {
            float v = kDual ? swiglu_f32(total, other) : total;
            if (residual) v += bf16_bits_to_f32(ptx::ld_global_dependent_u16(residual + n));
            out[n] = f32_to_bf16_bits(v);
        }
    }
}

constexpr int kGemvStageLimit = 104 * 1024;

// K parts per row: enough warps to keep the memory system busy when N is small.  Depends on
// (N, K) only, never on the number of activation rows.
inline int gemv_ksplit(int K, int N) {
    int ksplit = 1;
    const int slots = K >> 5;
    while (ksplit < 8 && (long)N * ksplit < 16384 && slots / (ksplit * 2) >= 16) ksplit *= 2;
    return ksplit;
}

template <int kM, bool kDual, int kStage>
inline int launch_gemv_instance(const uint16_t* x, GemvWeights a, GemvWeights b, const uint16_t* residual,
                                uint16_t* out, int K, int N, int sm_count, cudaStream_t stream) {
    constexpr int kRows = kDual ? (kM <= 2 ? 2 : 1) : (kM <= 2 ? 4 : (kM <= 4 ? 2 : 1));
    constexpr int kWarps = 8;
    auto kernel = affine_gemv_kernel<kM, kRows, kDual, kStage>;
    const int smem = kStage == kStageF32 ? gemv_f32_stage_bytes(K) : kStage == kStageBf16 ? kM * K * 2 : 0;
    if (smem > 32 * 1024) {  // the static partial-sum array counts toward the 48 KB default limit too
        static bool configured[64] = {};
        int device = 0;
        cudaGetDevice(&device);
        if (device >= 64 || !configured[device]) {
            if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kGemvStageLimit) != cudaSuccess)
                return MT_ERR_LAUNCH;
            if (device < 64) configured[device] = true;
        }
    }
    const int ksplit = gemv_ksplit(K, N);
    const int rows_per_cta = (kWarps / ksplit) * 2 * kRows;
    int grid = (N + rows_per_cta - 1) / rows_per_cta;
    // Resident CTAs per SM (each loops over its share of the rows): three when registers (80 x 256
    // threads) and the staged activations allow, else two.  The kernel waits on HBM latency with one
    // request in flight per lane and stream, so more resident warps mean more bytes in flight.
    const int cap = sm_count * (kM == 1 && smem <= 72 * 1024 ? 3 : 2);
    if (grid > cap) grid = cap;
    cudaLaunchConfig_t config = {};
    config.gridDim = dim3(grid, 1, 1);
    config.blockDim = dim3(kWarps * 32, 1, 1);
    config.dynamicSmemBytes = smem;
    config.stream = stream;
    cudaLaunchAttribute attrs[1];
    attrs[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attrs[0].val.programmaticStreamSerializationAllowed = 1;
    config.attrs = attrs;
    config.numAttrs = 1;
    return cudaLaunchKernelEx(&config, kernel, x, a, b, residual, out, K, N, ksplit) == cudaSuccess ? MT_OK
                                                                                                     : MT_ERR_LAUNCH;
}

constexpr int kGemvRingLimit = 112 * 1024;  // two CTAs per SM

// Where the rings serve: table words are copied whole, so tables start on one; byte offsets are 32 bits wide; the fp32
// activations of a row have the room that two CTAs' rings leave (K up to 13824), and a half-warp's rows exist.
// Everything else takes the register form below.
template <bool kDual>
inline bool gemv_ring_applicable(const GemvWeights& a, const GemvWeights& b, int K, int N) {
    for (const GemvWeights* w : {&a, &b})
        if (!aligned_to(w->scales, 4) || !aligned_to(w->biases, 4)) return false;
    return N >= kGemvRingRows && (long)N * (K >> 1) < (1l << 32) && gemv_f32_stage_bytes(K) + kGemvRingBytes <= kGemvRingLimit;
}

template <bool kDual>
inline int launch_gemv_ring(const uint16_t* x, GemvWeights a, GemvWeights b, const uint16_t* residual, uint16_t* out, int K,
                            int N, int sm_count, cudaStream_t stream) {
    static bool configured[64] = {};
    int device = 0;
    cudaGetDevice(&device);
    if (device >= 64 || !configured[device]) {
        if (cudaFuncSetAttribute(affine_gemv_ring_kernel<kDual>, cudaFuncAttributeMaxDynamicSharedMemorySize, kGemvRingLimit) != cudaSuccess)
            return MT_ERR_LAUNCH;
        if (device < 64) configured[device] = true;
    }
    const int ksplit = gemv_ksplit(K, N);
    const int rows_per_cta = 8 / ksplit * 2 * (kGemvRingRows / (kDual ? 2 : 1));
    const int grid = std::min((N + rows_per_cta - 1) / rows_per_cta, 2 * sm_count);
    cudaLaunchConfig_t config = {};
    config.gridDim = dim3(grid, 1, 1);
    config.blockDim = dim3(256, 1, 1);
    config.dynamicSmemBytes = gemv_f32_stage_bytes(K) + kGemvRingBytes;
    config.stream = stream;
    cudaLaunchAttribute attrs[1];
    attrs[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attrs[0].val.programmaticStreamSerializationAllowed = 1;
    config.attrs = attrs;
    config.numAttrs = 1;
    return cudaLaunchKernelEx(&config, affine_gemv_ring_kernel<kDual>, x, a, b, residual, out, K, N, ksplit) == cudaSuccess
               ? MT_OK : MT_ERR_LAUNCH;
}

// Activations are staged in shared memory when they fit kGemvStageLimit, which leaves room for two
// CTAs per SM (one row as fp32: K up to 24576; more rows as bf16); larger problems read them from
// global memory.
template <int kM, bool kDual>
inline int launch_gemv_m(const uint16_t* x, GemvWeights a, GemvWeights b, const uint16_t* residual, uint16_t* out,
                         int K, int N, int sm_count, cudaStream_t stream) {
    if constexpr (kM == 1) {
        if (gemv_ring_applicable<kDual>(a, b, K, N))
            return launch_gemv_ring<kDual>(x, a, b, residual, out, K, N, sm_count, stream);
        if (gemv_f32_stage_bytes(K) <= kGemvStageLimit)
            return launch_gemv_instance<kM, kDual, kStageF32>(x, a, b, residual, out, K, N, sm_count, stream);
    }
    if ((long)kM * K * 2 <= kGemvStageLimit)
        return launch_gemv_instance<kM, kDual, kStageBf16>(x, a, b, residual, out, K, N, sm_count, stream);
    return launch_gemv_instance<kM, kDual, kStageNone>(x, a, b, residual, out, K, N, sm_count, stream);
}

template <bool kDual>
inline int launch_gemv(const void* x, GemvWeights a, GemvWeights b, const void* residual, void* out, int M, int K,
                       int N, int sm_count, cudaStream_t stream) {
    const uint16_t* xp = static_cast<const uint16_t*>(x);
    const uint16_t* rp = static_cast<const uint16_t*>(residual);
    uint16_t* op = static_cast<uint16_t*>(out);
    switch (M) {
        case 1: return launch_gemv_m<1, kDual>(xp, a, b, rp, op, K, N, sm_count, stream);
        case 2: return launch_gemv_m<2, kDual>(xp, a, b, rp, op, K, N, sm_count, stream);
        case 3: return launch_gemv_m<3, kDual>(xp, a, b, rp, op, K, N, sm_count, stream);
        case 4: return launch_gemv_m<4, kDual>(xp, a, b, rp, op, K, N, sm_count, stream);
        case 5: return launch_gemv_m<5, kDual>(xp, a, b, rp, op, K, N, sm_count, stream);
        case 6: return launch_gemv_m<6, kDual>(xp, a, b, rp, op, K, N, sm_count, stream);
        case 7: return launch_gemv_m<7, kDual>(xp, a, b, rp, op, K, N, sm_count, stream);
        case 8: return launch_gemv_m<8, kDual>(xp, a, b, rp, op, K, N, sm_count, stream);
        default: return MT_ERR_SHAPE;
    }
}

}  // namespace mt
