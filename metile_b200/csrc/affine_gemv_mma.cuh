// INT4 affine projection of ONE activation row on the warp-level tensor cores (mma.sync), weights never rounded.
//
// Computes what affine_gemv.cuh computes (kernels/affine_qmv.py:4-54, SwiGLU :204-208, residual :124-131).  On the CUDA cores
// a weight costs one byte-permute and one FMA, and a warp issues 117 instructions per 1024 weights: at 2048 -> 128256 that is
// 27 of the 38 us, with the bytes needing 23.  Here a nibble q becomes the exact bf16 number (q - 8) / 64 (nine instructions
// per word of eight), m16n8k16 products with fp32 accumulators add (q - 8) x / 64 over a quantisation group of 64 columns,
// and a group is folded into the fp32 sum as fma(scale, P, fma(bias + 8 scale, X / 64, acc)), X = sum of the group's x.
//
// The codes are centred for the accumulators' sake, which cut off what lies 2^23 below the largest product: with 128 + q (seven
// instructions) sums that cancel were off by 2.4e-5 of their size in an MLP's down projection at 2048 / 8192, all to one
// side, on the CUDA cores by 9e-7; with centred codes by 5e-8.  2048 -> 128256 33.2 us (33.5 with 128 + q), MLP 2048 / 8192 13.2 (13.0).
//
// One activation row leaves seven of the product's eight columns over.  They hold eight GROUPS: column n of the B operand is
// x of group n of an item of eight.  Of an A operand, lanes t = 0, 1 of a row carry the two halves of group 2i and lanes t =
// 2, 3 those of group 2i + 1 (so a lane reads four words with one 16-byte load), and B is zero where the column's parity is
// not the lanes'.  Eight products make the sums of both groups, in columns 2i and 2i + 1, which are lane t = i's: it
// reads the scales of just those two groups, and nothing is multiplied, read or exchanged twice.
//
// A tile of 16 outputs belongs to a team of `parts` warps that share its K range; teams and CTAs take the tiles in turn.
// Items (16 rows x 512 columns, 4 KB) come by TMA into a ring of the warp's, one ahead of the one being read and the first before
// the wait for the preceding kernel; the tables of a tile's rows are one piece of memory and come by bulk copies.  The order of
// the sums is a function of (K, N, device).
#pragma once

#include <algorithm>

#include "affine_gemv.cuh"
#include "affine_umma.cuh"

namespace mt {

constexpr int kOneRowWarps = 8;
constexpr int kOneRowDepth = 2;        // ring items of a warp: one being read, one on its way
constexpr int kOneRowTables = 2;       // tiles whose tables a team holds
constexpr int kOneRowItemGroups = 8;
constexpr int kOneRowItemBytes = 16 * kOneRowItemGroups * 32;
constexpr float kOneRowUnit = 1.0f / 64.0f;  // of the sums, which are of w / 64 (see unpack_word_centred64)
constexpr int kOneRowSmemLimit = 224 * 1024;
constexpr int kOneRowSmemTwo = 110 * 1024;  // two CTAs per SM

enum : unsigned int { kWaitOneRowItem = 0x131, kWaitOneRowTables = 0x132 };

struct OneRowParams {
    CUtensorMap w_map[2];  // packed weights, uint32 [N, K/8], box {32, 16}: 128 bytes of sixteen rows, 128-byte swizzle
    const uint16_t* x;
    const uint16_t* scales[2];
    const uint16_t* biases[2];
    const uint16_t* residual;
    uint16_t* out;
    int K, N;
    int parts;        // warps of a team
    int table_bytes;  // of the scales (and of the biases) of sixteen rows
};

// The weight row of lane group g (and 8 + it): neighbouring groups, whose reads go together, take rows four apart, which the
// swizzle puts into the two halves of the banks.
__device__ __forceinline__ int one_row_tile_row(int g) { return (g >> 1) + 4 * (g & 1); }

// This lane's words of an item: of row tile_row and of the eighth row after it, of groups t / 2, 2 + t / 2, ...
__device__ __forceinline__ void one_row_words(const uint8_t* words, int tile_row, int t, uint32_t (&row)[4][4], uint32_t (&row8)[4][4]) {
    const uint32_t word_lane = (uint32_t)tile_row * 128u + ((uint32_t)(t ^ tile_row) << 4);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const uint8_t* at = words + (i >> 1) * 2048 + (word_lane ^ (uint32_t)((i & 1) << 6));
        const uint4 lo = *reinterpret_cast<const uint4*>(at), hi = *reinterpret_cast<const uint4*>(at + 1024);
        row[i][0] = lo.x; row[i][1] = lo.y; row[i][2] = lo.z; row[i][3] = lo.w;
        row8[i][0] = hi.x; row8[i][1] = hi.y; row8[i][2] = hi.z; row8[i][3] = hi.w;
    }
}

// Sums of (q - 8) / 64 x over groups 2t and 2t + 1 of the item: own[0], own[1] of this lane's row, own[2], own[3] of the eighth
// row after it.
__device__ __forceinline__ void one_row_products(const uint32_t (&row)[4][4], const uint32_t (&row8)[4][4], const uint32_t (&xr)[16], int t,
                                                 float (&own)[4]) {
    float sum[4][4] = {};
#pragma unroll
    for (int u = 0; u < 4; ++u)  // four chains side by side
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            uint32_t a[4], b[4];
            unpack_word_centred64(row[i][u], a);
            unpack_word_centred64(row8[i][u], b);
            ptx::mma_bf16_m16n8k16(sum[i], a[0], b[0], a[1], b[1], xr[4 * u], xr[4 * u + 1]);
            ptx::mma_bf16_m16n8k16(sum[i], a[2], b[2], a[3], b[3], xr[4 * u + 2], xr[4 * u + 3]);
        }
#pragma unroll
    for (int e = 0; e < 4; ++e) {
        const float low = t & 1 ? sum[1][e] : sum[0][e], high = t & 1 ? sum[3][e] : sum[2][e];
        own[e] = t & 2 ? high : low;
    }
}

template <bool kDual>
__global__ void __launch_bounds__(kOneRowWarps * 32, 2) affine_gemv_mma_kernel(const __grid_constant__ OneRowParams p) {
    constexpr int kStreams = kDual ? 2 : 1;
    extern __shared__ uint8_t one_row_smem[];
    __shared__ uint64_t item_full[kOneRowWarps][kOneRowDepth], table_full[kOneRowWarps][kOneRowTables];
    __shared__ float partial[2][kOneRowWarps][kStreams][16];
    __shared__ int abort_flag;

    const int warp = __shfl_sync(0xFFFFFFFFu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    const int warps = blockDim.x >> 5, parts = p.parts, teams = warps / parts;
    const int team = warp / parts, part = warp - team * parts;
    const int groups = p.K >> 6, chunks = (groups + kOneRowItemGroups - 1) / kOneRowItemGroups;
    const int begin = chunks * part / parts, end = chunks * (part + 1) / parts;
    const int tasks = (p.N + 15) >> 4, stride = teams * gridDim.x, first_task = team * gridDim.x + blockIdx.x;
    uint8_t* smem = one_row_smem + ((1024u - (ptx::smem_u32(one_row_smem) & 1023u)) & 1023u);
    uint8_t* ring = smem + warp * (kOneRowDepth * kOneRowItemBytes);
    uint8_t* x_tile = smem + warps * (kOneRowDepth * kOneRowItemBytes);  // 128 bytes per group
    float* x_sums = reinterpret_cast<float*>(x_tile + chunks * kOneRowItemGroups * 128);
    uint8_t* tables = reinterpret_cast<uint8_t*>(x_sums) + chunks * kOneRowItemGroups * 4 + team * (kOneRowTables * 2 * kStreams) * p.table_bytes;

    if (threadIdx.x == 0) {
        for (int w = 0; w < kOneRowWarps; ++w) {
            for (int i = 0; i < kOneRowDepth; ++i) ptx::mbar_init(&item_full[w][i], 1);
            for (int i = 0; i < kOneRowTables; ++i) ptx::mbar_init(&table_full[w][i], 1);
        }
        abort_flag = 0;
        ptx::mbar_fence_init();
    }
    __syncthreads();

    // ---- the copies of this warp's items, and of its team's tables (the first warp of a team)
    int copy_task = first_task, copy_chunk = begin, copy_stream = 0, table_task = first_task, table_slot = 0;
    // What was read in the slot, with ordinary loads, lies before the warp's last synchronisation and a proxy fence of every lane.
    auto copy_next = [&](int slot) {
        if (copy_task < tasks && ptx::elect_one()) {
            uint8_t* to = ring + slot * kOneRowItemBytes;
            ptx::mbar_expect_tx(&item_full[warp][slot], kOneRowItemBytes);
#pragma unroll
            for (int i = 0; i < 2; ++i)  // what lies past the end of the matrix is filled with zeros
                ptx::tma_load_2d(to + i * 2048, &p.w_map[copy_stream], copy_chunk * 64 + i * 32, copy_task * 16, &item_full[warp][slot]);
        }
        __syncwarp();
        if (kDual && copy_stream == 0) {
            copy_stream = 1;
            return;
        }
        copy_stream = 0;
        if (++copy_chunk == end) {
            copy_chunk = begin;
            copy_task += stride;
        }
    };
    // What the rows of the last tile leave over after whole 16 bytes is copied by a lane.
    auto copy_tables = [&] {
        if (part == 0 && table_task < tasks && ptx::elect_one()) {
            uint64_t* bar = &table_full[team][table_slot];
            uint8_t* to = tables + table_slot * (2 * kStreams) * p.table_bytes;
            const int n0 = table_task * 16, entries = min(16, p.N - n0) * groups, whole = entries & ~7;
            auto each = [&](auto&& copy) {
#pragma unroll
                for (int i = 0; i < 2 * kStreams; ++i) copy(to + i * p.table_bytes, ((i & 1) ? p.biases : p.scales)[i >> 1] + (size_t)n0 * groups);
            };
            if (whole < entries)
                each([&](uint8_t* at, const uint16_t* from) {
                    for (int e = whole; e < entries; ++e) reinterpret_cast<uint16_t*>(at)[e] = from[e];
                });
            ptx::mbar_expect_tx(bar, 4u * kStreams * whole);
            if (whole) each([&](uint8_t* at, const uint16_t* from) { ptx::bulk_load(at, from, 2u * whole, bar); });
        }
        __syncwarp();
        table_task += stride;
        table_slot = table_slot + 1 == kOneRowTables ? 0 : table_slot + 1;
    };

    ptx::griddep_launch_dependents();
#pragma unroll
    for (int i = 0; i < kOneRowTables; ++i) copy_tables();
#pragma unroll
    for (int i = 0; i < kOneRowDepth - 1; ++i) copy_next(i);
    ptx::griddep_wait();  // activations and residual are the preceding kernel's output
    // Eight activations per thread and pass: a word's pairs (x_i, x_i+4), and with its neighbours the sum of a group.
    for (int v = threadIdx.x; v < chunks * (kOneRowItemGroups * 8); v += blockDim.x) {
        uint4 raw = make_uint4(0u, 0u, 0u, 0u);
        if (v * 8 < p.K) raw = ptx::ld_global_dependent_u4(p.x + (size_t)v * 8);
        *reinterpret_cast<uint4*>(x_tile + v * 16) = make_uint4(__byte_perm(raw.x, raw.z, 0x5410), __byte_perm(raw.x, raw.z, 0x7632),
                                                                __byte_perm(raw.y, raw.w, 0x5410), __byte_perm(raw.y, raw.w, 0x7632));
        float sum = ((bf16_lo(raw.x) + bf16_hi(raw.x)) + (bf16_lo(raw.y) + bf16_hi(raw.y))) +
                    ((bf16_lo(raw.z) + bf16_hi(raw.z)) + (bf16_lo(raw.w) + bf16_hi(raw.w)));
#pragma unroll
        for (int offset = 1; offset < 8; offset <<= 1) sum += __shfl_xor_sync(0xFFFFFFFFu, sum, offset);
        if ((v & 7) == 0) x_sums[v >> 3] = kOneRowUnit * sum;
    }
    __syncthreads();

    const int tile_row = one_row_tile_row(g);
    const bool carries = (g & 1) == (t >> 1);  // whether this lane's column belongs to its half of the pairs
    const uint8_t* x_lane = x_tile + g * 128 + (t & 1) * 64;
    uint32_t xr[16];
    int loaded = -1;
    bool alive = true;
    int slot = 0, tile_slot = 0, parity = 0;
    uint32_t item_phase = 0, table_phase = 0;  // a bit per slot
    for (int task = first_task; task < tasks; task += stride, parity ^= 1) {
        const int n0 = task * 16;
        if (alive) alive = __all_sync(0xFFFFFFFFu, ptx::mbar_wait(&table_full[team][tile_slot], (table_phase >> tile_slot) & 1u, &abort_flag, kWaitOneRowTables));
        table_phase ^= 1u << tile_slot;
        const uint8_t* tile_tables = tables + tile_slot * (2 * kStreams) * p.table_bytes;
        tile_slot = tile_slot + 1 == kOneRowTables ? 0 : tile_slot + 1;
        float acc[kStreams][2] = {};
        for (int chunk = begin; chunk < end; ++chunk) {
            if (chunk != loaded) {
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    const uint4 v = carries ? *reinterpret_cast<const uint4*>(x_lane + chunk * 1024 + u * 16) : make_uint4(0u, 0u, 0u, 0u);
                    xr[4 * u] = v.x; xr[4 * u + 1] = v.y; xr[4 * u + 2] = v.z; xr[4 * u + 3] = v.w;
                }
                loaded = chunk;
            }
            const int group = chunk * kOneRowItemGroups + 2 * t;  // this lane's two
            const float2 xs = *reinterpret_cast<const float2*>(x_sums + group);
#pragma unroll
            for (int s = 0; s < kStreams; ++s) {
                if (alive) alive = __all_sync(0xFFFFFFFFu, ptx::mbar_wait(&item_full[warp][slot], (item_phase >> slot) & 1u, &abort_flag, kWaitOneRowItem));
                item_phase ^= 1u << slot;
                ptx::fence_proxy_async_smem();  // the slot that was read before this one is filled again
                __syncwarp();
                copy_next(slot == 0 ? kOneRowDepth - 1 : slot - 1);
                const uint8_t* words = ring + slot * kOneRowItemBytes;
                if (++slot == kOneRowDepth) slot = 0;
                uint32_t row[4][4], row8[4][4];
                one_row_words(words, tile_row, t, row, row8);
                float own[4];
                one_row_products(row, row8, xr, t, own);
                const uint16_t* scale_row = reinterpret_cast<const uint16_t*>(tile_tables + 2 * s * p.table_bytes);
                const uint16_t* bias_row = reinterpret_cast<const uint16_t*>(tile_tables + (2 * s + 1) * p.table_bytes);
#pragma unroll
                for (int r = 0; r < 2; ++r)
#pragma unroll
                    for (int e = 0; e < 2; ++e) {
                        if (group + e >= groups) continue;
                        const int at = (tile_row + 8 * r) * groups + group + e;
                        const float scale = bf16_bits_to_f32(scale_row[at]), centre = fmaf(8.0f, scale, bf16_bits_to_f32(bias_row[at]));
                        acc[s][r] = fmaf(scale, own[2 * r + e], fmaf(centre, e ? xs.y : xs.x, acc[s][r]));
                    }
            }
        }

        // ---- the lanes' and the warps' parts; lane t = 0 goes on with row g, lane t = 1 with row g + 8
        float total[kStreams];
#pragma unroll
        for (int s = 0; s < kStreams; ++s) {
#pragma unroll
            for (int r = 0; r < 2; ++r) {
                acc[s][r] += __shfl_xor_sync(0xFFFFFFFFu, acc[s][r], 1);
                acc[s][r] += __shfl_xor_sync(0xFFFFFFFFu, acc[s][r], 2);
            }
            total[s] = (t == 0 ? acc[s][0] : acc[s][1]) / kOneRowUnit;
        }
        const int row = tile_row + 8 * (t & 1), n = n0 + row;
        const bool finishes = part == 0 && t < 2 && n < p.N;
        const uint32_t extra = !kDual && p.residual && finishes ? ptx::ld_global_dependent_u16(p.residual + n) : 0u;
        ptx::fence_proxy_async_smem();  // the tables are filled again
        if (parts > 1) {
            if (t < 2) {
#pragma unroll
                for (int s = 0; s < kStreams; ++s) partial[parity][warp][s][row] = total[s];
            }
            ptx::named_barrier_sync(1 + team, parts * 32);
            if (part == 0) {
#pragma unroll
                for (int s = 0; s < kStreams; ++s)
                    for (int w = 1; w < parts; ++w) total[s] += partial[parity][warp + w][s][row];
            }
        } else {
            __syncwarp();
        }
        if (finishes) p.out[n] = f32_to_bf16_bits(kDual ? swiglu_f32(total[0], total[kStreams - 1]) : total[0] + bf16_bits_to_f32(extra));
        copy_tables();
    }
    if (abort_flag) ptx::drain_copies();
}

// ------------------------------------------------------------------------------- host side
struct OneRowPlan {
    int parts, teams, grid, table_bytes, smem;
};

// Warps per team and teams per CTA: what finishes the tiles soonest, in us, fitted to all splits of 72 shapes in replayed graphs (what
// it picks takes 4 % longer than the best split on average).  An item takes a warp 0.43 us (0.61 where one warp walks along the
// rows alone) or 0.47 and 0.022 for each busy warp of its SM; a team of several warps meets once per tile.  Two items in a ring
// and two tiles' tables are best or within 2 % nearly everywhere (2048 -> 128256 29.0 us; three items, which leave room for one
// CTA per SM, 32.6; the tables requested when their tile begins 30.4).
inline bool one_row_plan(OneRowPlan& best, int K, int N, bool dual, int sm_count) {
    static const int splits[11][2] = {{1, 8}, {1, 6}, {2, 4}, {2, 3}, {2, 2}, {3, 2}, {3, 1}, {4, 2}, {4, 1}, {6, 1}, {8, 1}};
    const int groups = K / 64, chunks = (groups + kOneRowItemGroups - 1) / kOneRowItemGroups, tasks = (N + 15) / 16;
    const int streams = dual ? 2 : 1;
    double best_cost = -1.0;
    for (const auto& split : splits) {
        OneRowPlan plan;
        const int parts = plan.parts = split[0];
        plan.teams = split[1];
        if (parts > chunks) continue;
        plan.table_bytes = (16 * groups * 2 + 127) / 128 * 128;
        plan.smem = 1024 + parts * plan.teams * kOneRowDepth * kOneRowItemBytes + chunks * kOneRowItemGroups * (128 + 4) +
                    plan.teams * kOneRowTables * 2 * streams * plan.table_bytes;
        if (plan.smem > kOneRowSmemLimit) continue;
        const int resident = plan.smem <= kOneRowSmemTwo ? 2 : 1;
        plan.grid = std::min((tasks + plan.teams - 1) / plan.teams, resident * sm_count);
        const int slots = plan.teams * plan.grid, waves = (tasks + slots - 1) / slots, steps = (chunks + parts - 1) / parts;
        const double busy = parts * plan.teams * ((plan.grid + sm_count - 1) / sm_count) * (double)chunks / (steps * parts);
        const double item = std::max(parts == 1 ? 0.61 : 0.43, 0.47 + 0.022 * busy);
        const double even = (double)tasks / slots, turns = even <= 1.0 ? 1.0 : 0.62 * waves + 0.38 * even;
        const double cost = turns * (steps * streams * item + (parts > 1 ? 0.036 * parts : 0.0) + 0.012 * streams);
        if (best_cost >= 0 && cost >= best_cost) continue;
        best_cost = cost;
        best = plan;
    }
    return best_cost >= 0;
}

// Where it is used: tables that bulk copies take, items that are not mostly empty, and weights enough: below, both forms take a
// few us (with codes of 128 + q, here | with the rings of affine_gemv.cuh: 1024 -> 6544 3.5 | 2.9, 2048 -> 157 2.5 | 2.0; gate|up in an MLP 1088 / 4096
// 9.4 | 7.4, 1536 / 5248 10.8 | 10.7, 1920 / 5056 10.5 | 11.0).  A long K range with few tiles takes more of them to pay (4096
// -> 4096 4.5 | 4.4, 8192 -> 2048 5.7 | 4.9; down in an MLP 3584 / 12288 24.1 | 24.2, 3008 / 17024 30.0 | 32.7).
inline bool one_row_applicable(const GemvWeights& a, const GemvWeights& b, int K, int N, bool dual) {
    const int groups = K / 64, chunks = (groups + kOneRowItemGroups - 1) / kOneRowItemGroups;
    for (const GemvWeights* w : {&a, &b})
        if (!aligned_to(w->scales, 16) || !aligned_to(w->biases, 16)) return false;
    if (10 * kOneRowItemGroups * chunks > 18 * groups) return false;
    const double weights = (double)N * K * (dual ? 2 : 1);
    return weights >= (dual ? 18e6 : chunks <= 3 ? 8e6 : chunks <= 5 ? 11e6 : 45e6);
}

// And where the plan leaves too much of the chip idle, the rings are faster (here | there, us, in replayed graphs; of 1090 random
// shapes of one row above the sizes above 66 took more than 2 % longer here, to 33 %, and with these rules 8, to 13 %):
//   two matrices and few tiles                          7104 -> 1312 8.3 | 6.4, 12928 -> 775 11.2 | 8.4
//   a second step that few of a team's warps have, on a part of the SMs    3520 -> 2688 7.8 | 6.3, 7232 -> 1920 9.0 | 8.5
//   tiles for just more than one turn of six-warp teams, along a long row  10240 -> 5120 20.2 | 17.4, 13632 -> 5056 16.7 | 15.6
//   several turns of small teams, six warps to a CTA    832 -> 19255 8.9 | 8.3, 768 -> 24293 10.2 | 9.5
inline bool one_row_pays(const OneRowPlan& plan, int K, int N, bool dual, int sm_count) {
    const int chunks = (K / 64 + kOneRowItemGroups - 1) / kOneRowItemGroups, tiles = (N + 15) / 16, warps = plan.parts * plan.teams;
    const double turns = (double)tiles / (plan.teams * plan.grid);
    if (K > 13824) return true;  // the rings do not serve it
    if (plan.parts == 6 && turns > 1.0 && turns < 1.12) return false;
    if (!dual) return true;
    if (tiles < 0.7 * sm_count) return false;
    if (warps == 8 && plan.parts < chunks && chunks < 2 * plan.parts && plan.grid < 0.945 * sm_count) return false;
    return !(warps == 6 && plan.parts == chunks && chunks > 1 && turns > 1.3);
}

template <bool kDual>
inline int launch_one_row(const void* x, const GemvWeights& a, const GemvWeights& b, const void* residual, void* out, int K, int N,
                          const OneRowPlan& plan, cudaStream_t stream) {
    static bool configured[64] = {};
    int device = 0;
    cudaGetDevice(&device);
    if (device >= 64 || !configured[device]) {
        if (cudaFuncSetAttribute(affine_gemv_mma_kernel<kDual>, cudaFuncAttributeMaxDynamicSharedMemorySize, kOneRowSmemLimit) != cudaSuccess)
            return MT_ERR_LAUNCH;
        if (device < 64) configured[device] = true;
    }
    OneRowParams params;
    if (!encode_weight_map(&params.w_map[0], a.w, K, N, 16)) return MT_ERR_LAUNCH;
    if (kDual && !encode_weight_map(&params.w_map[1], b.w, K, N, 16)) return MT_ERR_LAUNCH;
    params.x = static_cast<const uint16_t*>(x);
    params.scales[0] = a.scales;
    params.scales[1] = b.scales;
    params.biases[0] = a.biases;
    params.biases[1] = b.biases;
    params.residual = static_cast<const uint16_t*>(residual);
    params.out = static_cast<uint16_t*>(out);
    params.K = K;
    params.N = N;
    params.parts = plan.parts;
    params.table_bytes = plan.table_bytes;
    cudaLaunchConfig_t config = {};
    config.gridDim = dim3(plan.grid, 1, 1);
    config.blockDim = dim3(plan.parts * plan.teams * 32, 1, 1);
    config.dynamicSmemBytes = plan.smem;
    config.stream = stream;
    cudaLaunchAttribute attrs[1];
    attrs[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attrs[0].val.programmaticStreamSerializationAllowed = 1;
    config.attrs = attrs;
    config.numAttrs = 1;
    return cudaLaunchKernelEx(&config, affine_gemv_mma_kernel<kDual>, params) == cudaSuccess ? MT_OK : MT_ERR_LAUNCH;
}

}  // namespace mt
