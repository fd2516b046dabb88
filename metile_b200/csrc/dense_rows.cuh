// Dense bf16 small-batch projection: rows of a batch share every weight load, and each row's
// result is bit-identical to running that row alone.
//
// Follows the arithmetic order of the reference's generated small-batch kernels
// (metile/compiler/dense.py:193-381, emitted by metile/codegen/msl_emitter.py:1067-1120 and
// :1218-1251): lane l of a 32-lane group owns k = 128*b + 4*l .. +3, accumulates in fp32 in
// ascending (b, component) order with fused multiply-adds, lanes are combined by a shuffle-down
// tree with offsets 16, 8, 4, 2, 1, lane 0 rounds to bf16, then the typed epilogue runs:
//   residual : bf16(bf16(acc) + residual)
//   SwiGLU   : l = bf16(gate), r = bf16(up), y = 1/(1+exp(|l|)), sig = bf16(l<0 ? y : 1-y),
//              out = bf16(bf16(l*sig) * r)
// One warp produces kOut outputs for all rows of a chunk of up to 16; a launch holds up to 37 chunks (of 148 SMs).
// What bounds it: one to four rows the weights' bytes (K = 4096, N = 12000, one row: 20.9 us, 4.7 TB/s; with weights
// requested into registers 24.8), more rows the multiply-adds, whose order leaves no room for tensor cores,
// together with the conversions between them (128 rows of 1536 -> 8960: 98 us, half of the FMA rate; one
// launch per 16 rows, two outputs per warp and activations read through L1: 248).  16 rows of that shape 32.9 -> 15.3.
#pragma once

#include <algorithm>

#include "common.cuh"
#include "ptx.cuh"

namespace mt {

__device__ __forceinline__ float round_bf16(float v) { return bf16_bits_to_f32(f32_to_bf16_bits(v)); }

enum class DenseEpilogue { kPlain, kSwiglu };

// The shuffle-down tree of kN values at once: at every offset a lane keeps the half of the values that its bit of
// the offset names and adds the other lane's copies of them, so 64 values take 62 exchanges instead of 320.  Which
// two partial sums are added, and when, is what the tree says; only the lane that ends up with a total differs.
template <int kN, int kOffset, int kSize>
__device__ __forceinline__ void fold_lanes(float (&v)[kSize], int lane) {
    if constexpr (kOffset > 0) {
        if constexpr (kN % 2 == 0) {
            const bool upper = lane & kOffset;
#pragma unroll
            for (int i = 0; i < kN / 2; ++i) {
                const float keep = upper ? v[i + kN / 2] : v[i], send = upper ? v[i] : v[i + kN / 2];
                v[i] = keep + __shfl_xor_sync(0xFFFFFFFFu, send, kOffset);
            }
            fold_lanes<kN / 2, kOffset / 2>(v, lane);
        } else {
#pragma unroll
            for (int i = 0; i < kN; ++i) v[i] += __shfl_xor_sync(0xFFFFFFFFu, v[i], kOffset);
            fold_lanes<kN, kOffset / 2>(v, lane);
        }
    }
}
// Where the totals are: a lane has folded_count<kN>() of them from value `first` on, if it is their owner.
template <int kN, int kOffset = 16>
__host__ __device__ constexpr int folded_count() {
    if constexpr (kOffset == 0) return kN;
    else return folded_count<kN % 2 == 0 ? kN / 2 : kN, kOffset / 2>();
}
template <int kN, int kOffset = 16>
__device__ __forceinline__ int folded_first(int lane, bool& owner) {
    if constexpr (kOffset == 0) return 0;
    else if constexpr (kN % 2 == 0) return (lane & kOffset ? kN / 2 : 0) + folded_first<kN / 2, kOffset / 2>(lane, owner);
    else {
        if (lane & kOffset) owner = false;
        return folded_first<kN, kOffset / 2>(lane, owner);
    }
}

// One CTA of sixteen warps per SM.  Weights go through a private ring of each warp by asynchronous copies, 28 KB (one row of
// weights at a time) to 80 KB in flight per SM: requested into registers some blocks ahead they arrived one block at a time, since a
// warp's few scoreboards are shared by the blocks (1536 -> 8960, one row: 12.4 us, now 6.3).  No registers are
// spent on it, so a warp holds 64 accumulators, and an activation is read and converted once for four outputs.
constexpr int kDenseThreads = 512;
constexpr int kDenseWarps = kDenseThreads / 32;
// 128-column blocks of a warp's `streams` rows of weights that are in its ring, all but one of them in flight.
__host__ __device__ constexpr int dense_slots(int streams) { return streams >= 3 ? 6 : 8; }
__host__ __device__ constexpr int dense_ring_bytes(int streams) { return kDenseWarps * dense_slots(streams) * streams * 256; }
constexpr int kDenseSmemBytes = 227 * 1024;
// Activations are staged as pairs of rows: a single row takes the room of two.
constexpr long dense_smem_bytes(int m, int streams, int K) { return dense_ring_bytes(streams) + 2l * (m + m % 2) * K; }

struct DenseParams {
    const uint16_t *x, *w[2], *residual;
    uint16_t* out;
    int M, K, N;
    int chunk_rows;   // rows of a chunk, kM at most
    int chunk_ctas;   // CTAs of a chunk
    bool wide;        // the weights are 16-byte aligned
    bool staged;      // the activations fit shared memory (else kM is 1)
};

// kM: rows of a chunk, 1 or even (rows past the chunk's are computed on whatever is there and not stored).
template <int kM, int kOut, DenseEpilogue kEp>
__global__ void __launch_bounds__(kDenseThreads, 1) dense_rows_kernel(const __grid_constant__ DenseParams p) {
    static_assert(kM == 1 || kM % 2 == 0);
    constexpr int kStreams = kEp == DenseEpilogue::kSwiglu ? 2 : 1;
    constexpr int kPairs = (kM + 1) / 2, kRows = kStreams * kOut, kSlots = dense_slots(kRows);
    extern __shared__ __align__(16) uint8_t dense_smem[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint8_t* ring = dense_smem + warp * (kSlots * kRows * 256);
    uint2* x_words = reinterpret_cast<uint2*>(dense_smem + dense_ring_bytes(kRows));  // [128 columns][pair of rows][half of a lane's four][lane]: a word of each row
    const int chunk = blockIdx.x / p.chunk_ctas, cta = blockIdx.x - chunk * p.chunk_ctas;
    const int m0 = chunk * p.chunk_rows, rows = min(p.chunk_rows, p.M - m0);
    const int first_task = warp * p.chunk_ctas + cta;  // SM by SM: the tasks of a last round are spread
    const int tasks = (p.N + kOut - 1) / kOut, stride = kDenseWarps * p.chunk_ctas;
    const int blocks = p.K >> 7;
    const uint16_t* x = p.x + (size_t)m0 * p.K;

    // The copies run through all tasks of the warp without a break.  16 bytes per copy and lane, two rows at a time;
    // a row without a partner, or weights that are only 8-byte aligned, 8 bytes.
    int copy_task = first_task, copy_block = 0;
    auto copy_next = [&](int copy_slot) {
        if (copy_task < tasks) {
            const int n0 = min(copy_task * kOut, p.N - kOut);
            uint8_t* slot = ring + copy_slot * (kRows * 256);
#pragma unroll
            for (int r = 0; r < kRows; ++r) {
                if (p.wide && r % 2 == 0 && r + 1 < kRows) {
                    const int row = r + (lane >> 4);
                    const bool second = kStreams == 2 && (kOut == 1 ? row == 1 : r >= kOut);
                    const uint16_t* from = p.w[second] + (size_t)(n0 + row - (second ? kOut : 0)) * p.K;
                    ptx::cp_async_16(slot + row * 256 + (lane & 15) * 16, from + copy_block * 128 + (lane & 15) * 8);
                } else if (!p.wide || (r % 2 == 0 && r + 1 == kRows)) {
                    const uint16_t* from = p.w[kStreams == 2 && r >= kOut] + (size_t)(n0 + r % kOut) * p.K;
                    ptx::cp_async_8(slot + r * 256 + lane * 8, from + copy_block * 128 + lane * 4);
                }
            }
            if (++copy_block == blocks) copy_block = 0, copy_task += stride;
        }
        ptx::cp_async_commit();
    };
    ptx::griddep_launch_dependents();
    ptx::griddep_wait();
#pragma unroll
    for (int i = 0; i < kSlots - 1; ++i) copy_next(i);

    for (int i = threadIdx.x; i < (kM > 1 || p.staged ? kPairs * blocks * 32 : 0); i += kDenseThreads) {
        const int pair = i / (blocks * 32), at = i - pair * (blocks * 32);
        const uint2* from = reinterpret_cast<const uint2*>(x + (size_t)min(2 * pair, rows - 1) * p.K) + at;
        const uint2 a = *from, b = *(from + (2 * pair + 1 < rows ? p.K / 4 : 0));
        uint2* to = x_words + (at / 32 * kPairs + pair) * 64 + at % 32;
        to[0] = make_uint2(a.x, b.x);
        to[32] = make_uint2(a.y, b.y);
    }
    __syncthreads();

    int slot = 0;
    constexpr int kCount = folded_count<kOut * kM>();
    for (int task = first_task; task < tasks; task += stride) {
        const int n0 = min(task * kOut, p.N - kOut);  // the last task computes some of its neighbour's outputs again
        bool owner = true;
        const int first = folded_first<kOut * kM>(lane, owner);
        uint16_t extra[kCount];
        if (kEp == DenseEpilogue::kPlain && p.residual) {
#pragma unroll
            for (int i = 0; i < kCount; ++i) {
                const int m = (first + i) / kOut, n = n0 + (first + i) % kOut;
                extra[i] = m < rows ? p.residual[(size_t)(m0 + m) * p.N + n] : (uint16_t)0;
            }
        }
        float2 acc[kStreams][kOut][kPairs];
#pragma unroll
        for (int s = 0; s < kStreams; ++s)
#pragma unroll
            for (int o = 0; o < kOut; ++o)
#pragma unroll
                for (int j = 0; j < kPairs; ++j) acc[s][o][j] = make_float2(0.0f, 0.0f);

        for (int b = 0; b < blocks; ++b) {
            ptx::cp_async_wait_group<kSlots - 2>();
            __syncwarp();
            copy_next(slot == 0 ? kSlots - 1 : slot - 1);  // into the slot that was read before this one
            const uint8_t* tile = ring + slot * (kRows * 256);
            if (++slot == kSlots) slot = 0;
            uint2 words[kRows];
#pragma unroll
            for (int r = 0; r < kRows; ++r) words[r] = *reinterpret_cast<const uint2*>(tile + r * 256 + lane * 8);
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                float w[kRows][2];
#pragma unroll
                for (int r = 0; r < kRows; ++r) {
                    w[r][0] = bf16_lo(h ? words[r].y : words[r].x);
                    w[r][1] = bf16_hi(h ? words[r].y : words[r].x);
                }
#pragma unroll
                for (int j = 0; j < kPairs; ++j) {
                    uint2 xs;
                    if (kM > 1 || p.staged) xs = x_words[(b * kPairs + j) * 64 + h * 32 + lane];
                    else xs.x = reinterpret_cast<const uint32_t*>(x)[b * 64 + lane * 2 + h];
#pragma unroll
                    for (int c = 0; c < 2; ++c) {
                        const float2 x2 = c ? make_float2(bf16_hi(xs.x), bf16_hi(xs.y)) : make_float2(bf16_lo(xs.x), bf16_lo(xs.y));
#pragma unroll
                        for (int r = 0; r < kRows; ++r) {
                            float2& sum = acc[r / kOut][r % kOut][j];
                            if constexpr (kM == 1) sum.x = fmaf(w[r][c], x2.x, sum.x);
                            else sum = ptx::fma_f32x2(make_float2(w[r][c], w[r][c]), x2, sum);
                        }
                    }
                }
            }
        }

        float total[kStreams][kOut * kM];
#pragma unroll
        for (int s = 0; s < kStreams; ++s) {
#pragma unroll
            for (int o = 0; o < kOut; ++o)
#pragma unroll
                for (int m = 0; m < kM; ++m) total[s][m * kOut + o] = m % 2 ? acc[s][o][m / 2].y : acc[s][o][m / 2].x;
            fold_lanes<kOut * kM, 16>(total[s], lane);
        }
#pragma unroll
        for (int i = 0; i < kCount; ++i) {
            const int m = (first + i) / kOut, n = n0 + (first + i) % kOut;
            if (!owner || m >= rows || n < task * kOut) continue;
            float v;
            if constexpr (kEp == DenseEpilogue::kSwiglu) {
                const float left = round_bf16(total[0][i]);
                const float right = round_bf16(total[kStreams - 1][i]);
                const float y = 1.0f / (1.0f + expf(fabsf(left)));
                const float sigmoid = round_bf16(left < 0.0f ? y : 1.0f - y);
                v = round_bf16(left * sigmoid) * right;
            } else {
                v = round_bf16(total[0][i]);
                if (p.residual) v += bf16_bits_to_f32(extra[i]);
            }
            p.out[(size_t)(m0 + m) * p.N + n] = f32_to_bf16_bits(v);
        }
    }
}

template <int kM, int kOut, DenseEpilogue kEp>
inline int launch_dense_instance(DenseParams p, int chunks, int sm_count, int device, cudaStream_t stream) {
    static bool configured[64] = {};
    if (!(device < 64 && configured[device])) {
        if (cudaFuncSetAttribute(dense_rows_kernel<kM, kOut, kEp>, cudaFuncAttributeMaxDynamicSharedMemorySize, kDenseSmemBytes) != cudaSuccess)
            return MT_ERR_LAUNCH;
        if (device < 64) configured[device] = true;
    }
    p.chunk_ctas = std::min(std::max(sm_count / chunks, 1), (p.N + kOut - 1) / kOut);
    cudaLaunchConfig_t config = {};
    config.gridDim = dim3(chunks * p.chunk_ctas, 1, 1);
    config.blockDim = dim3(kDenseThreads, 1, 1);
    constexpr int kRows = kOut * (kEp == DenseEpilogue::kSwiglu ? 2 : 1);
    const long smem = dense_smem_bytes(kM, kRows, p.K);
    p.staged = smem <= kDenseSmemBytes;
    config.dynamicSmemBytes = p.staged ? smem : dense_ring_bytes(kRows);
    config.stream = stream;
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    config.attrs = &attr;
    config.numAttrs = 1;
    return cudaLaunchKernelEx(&config, dense_rows_kernel<kM, kOut, kEp>, p) == cudaSuccess ? MT_OK : MT_ERR_LAUNCH;
}

template <int kM, DenseEpilogue kEp>
inline int launch_dense_m(int outs, const DenseParams& p, int chunks, int sm_count, int device, cudaStream_t stream) {
    if (outs == 1) return launch_dense_instance<kM, 1, kEp>(p, chunks, sm_count, device, stream);
    if (outs == 2) return launch_dense_instance<kM, 2, kEp>(p, chunks, sm_count, device, stream);
    if constexpr (kEp == DenseEpilogue::kPlain) {
        if (outs == 3) return launch_dense_instance<kM, 3, kEp>(p, chunks, sm_count, device, stream);
        if (outs == 4) return launch_dense_instance<kM, 4, kEp>(p, chunks, sm_count, device, stream);
    }
    return MT_ERR_SHAPE;
}

constexpr int kDenseRows[] = {1, 2, 4, 8, 12, 16};

// Cycles of a launch over `chunks` chunks with room for m rows and `outs` outputs per warp: rounds of tasks, bound by
// issue (what a warp's block takes) or by the latency of a warp alone, or the reading of the matrix, of which
// the chunks after the first find most in L2; and before them the activations' way to shared memory.  Fitted to 1 to
// 128 rows of 256 to 12000 outputs.  Few outputs make small chunks the better choice (16 rows, 4096 -> 256: 12.6 us,
// 43 in one chunk).
inline long dense_cost(int m, int outs, int streams, int chunks, int K, int N, int sm_count) {
    const int ctas = std::max(sm_count / chunks, 1), blocks = K / 128, rows = streams * outs;
    const int tasks = ((N + outs - 1) / outs + ctas - 1) / ctas, rounds = tasks / kDenseWarps, rest = tasks % kDenseWarps;
    const long warp = (long)blocks * (rows * 4 * m + 5 * m + 60), alone = (long)blocks * (rows * 4 * m + 5 * m + 200);
    const long math = rounds * std::max(4 * warp, alone) + (rest ? std::max((rest + 3) / 4 * warp, alone) : 0) + (rounds + (rest > 0)) * 400;
    const long read = (long)N * K / 2650 * streams * (chunks + 1) / 2;
    return std::max(math, read) + (long)m * K / 20 + 2000;
}

template <DenseEpilogue kEp>
inline int launch_dense(const void* x, const void* w0, const void* w1, const void* residual, void* out, int M, int K,
                        int N, int sm_count, cudaStream_t stream) {
    if (M < 1 || K < 128 || K % 128 || N < 1) return MT_ERR_SHAPE;
    if (!aligned_to(x, 8) || !aligned_to(w0, 8) || (w1 && !aligned_to(w1, 8))) return MT_ERR_ALIGN;
    int device = 0;
    if (cudaGetDevice(&device) != cudaSuccess) return MT_ERR_DEVICE;
    DenseParams p = {};
    p.w[0] = static_cast<const uint16_t*>(w0);
    p.w[1] = static_cast<const uint16_t*>(w1);
    p.K = K;
    p.N = N;
    p.wide = aligned_to(w0, 16) && aligned_to(w1, 16);
    constexpr int kStreams = kEp == DenseEpilogue::kSwiglu ? 2 : 1;
    const int launch_chunks = std::max(sm_count / 4, 1);  // of one launch
    int room = 0, outs = 1;
    long best = 0;
    for (int m : kDenseRows) {
        const int chunks = (M + m - 1) / m, launches = (chunks + launch_chunks - 1) / launch_chunks;
        for (int streams = kStreams; streams <= 4; streams += kStreams) {
            if (streams / kStreams > N || (m > 1 && dense_smem_bytes(m, streams, K) > kDenseSmemBytes)) continue;
            const long cost = launches * dense_cost(m, streams / kStreams, kStreams, std::min(chunks, launch_chunks), K, N, sm_count);
            if (room == 0 || cost < best) best = cost, room = m, outs = streams / kStreams;
        }
        if (m >= M) break;
    }
    for (int m0 = 0; m0 < M; m0 += launch_chunks * room) {
        p.M = std::min(M - m0, launch_chunks * room);
        const int chunks = (p.M + room - 1) / room;
        p.chunk_rows = (p.M + chunks - 1) / chunks;
        p.x = static_cast<const uint16_t*>(x) + (size_t)m0 * K;
        p.residual = residual ? static_cast<const uint16_t*>(residual) + (size_t)m0 * N : nullptr;
        p.out = static_cast<uint16_t*>(out) + (size_t)m0 * N;
        const int used = (p.M + p.chunk_rows - 1) / p.chunk_rows;
        int rc;
        switch (room) {
            case 1: rc = launch_dense_m<1, kEp>(outs, p, used, sm_count, device, stream); break;
            case 2: rc = launch_dense_m<2, kEp>(outs, p, used, sm_count, device, stream); break;
            case 4: rc = launch_dense_m<4, kEp>(outs, p, used, sm_count, device, stream); break;
            case 8: rc = launch_dense_m<8, kEp>(outs, p, used, sm_count, device, stream); break;
            case 12: rc = launch_dense_m<12, kEp>(outs, p, used, sm_count, device, stream); break;
            default: rc = launch_dense_m<16, kEp>(outs, p, used, sm_count, device, stream); break;
        }
        if (rc != MT_OK) return rc;
    }
    return MT_OK;
}

}  // namespace mt
