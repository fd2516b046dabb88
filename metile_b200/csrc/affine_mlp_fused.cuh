// The whole INT4 affine MLP  out = down(silu(x Wg^T) * (x Wu^T)) + residual  for a handful of
// activation rows as ONE launch, one CTA per SM.  Two kernels share the launch structure:
// the one-row kernel described first (one to four rows, default for one) and the eight-column kernel
// further down (up to eight rows, default from two).
//
// Why one launch.  At a few rows the MLP is a pure stream of packed weights (28 MB at the
// Llama-3.2-1B shape: 4.4 us at the measured HBM rate), and two dependent kernels spend more time
// starting, ramping up their loads and draining than moving those bytes.  Here a CTA streams its rows
// of gate and up, then its rows of down, through rings of shared memory fed by bulk copies.
// HBM stays busy while the arithmetic runs behind the copies.  The two projections are separated by a meeting of all CTAs (every hidden
// activation must exist before any down row can be summed); down rows are already in the rings
// when it is over.
//
// Rows.  CTA c owns gate/up rows [c*I/grid, (c+1)*I/grid) and down rows [c*H/grid, (c+1)*H/grid).
//
// The one-row kernel multiplies as affine_gemv_mma.cuh does: mma.sync over units of 16 weight rows x 512
// columns, eight quantisation groups in the product's eight columns.  A CTA's rows are cut into as few
// tiles as sixteen rows allow, all of one height (55 gate rows: four of fourteen), a tile's K range into
// units, and unit u of the CTA belongs to warp u % 8: where a tile has no more than eight column units, a warp's are of the
// same columns throughout a projection, and its activations are read once, into registers.  Every warp
// has a ring of its own and issues its own copies; the tables of all rows of the CTA come by one copy each.  The units' sums of a
// row meet in shared memory and are added in column order: the fp32 order depends on (H, I) only.  More rows than one
// multiply the same words again.
//
// What bounds it (2048 / 8192): its start and end and the meeting of the CTAs, about 5 us, beside the bytes' 4.4.  Launch after
// launch, us, called from Python and in a replayed graph: byte-permutes and FMAs on the CUDA cores in a cooperative
// launch 16.4 and 15.1, products on mma.sync 16.2, an ordinary launch (fused_meet) of sixteen warps with all weights of a
// CTA on their way at once 13.2 and 15.3, eight warps and room for two CTAs per SM, so that the next launch begins its
// copies behind the meeting, 13.2 and 12.6 (with centred codes and small meeting slots, as now, 12.8 and 12.7).
#pragma once

#include <cuda.h>

#include "affine_gemv_mma.cuh"
#include "common.cuh"
#include "meeting_slots.h"
#include "ptx.cuh"

namespace mt {

constexpr int kFusedComputeWarps = 8;
constexpr int kFusedComputeThreads = kFusedComputeWarps * 32;
constexpr int kFusedThreads = kFusedComputeThreads + 32;  // + the producer warp
constexpr int kFusedOneWarps = 8;
constexpr int kFusedOneThreads = kFusedOneWarps * 32;
constexpr int kFusedMaxRows = 4;
// Rows the one-row kernel serves by default; two to four only when asked with MT_FLAG_MLP_FUSED.  The rule
// for one row is older than affine_gemv_mma.cuh and no longer the faster one everywhere: at hidden / intermediate widths of 1024 / 1024, 1024 /
// 4096, 2048 / 4096, 2048 / 8192, 4096 / 4096, 4096 / 8192 this kernel takes 6.2 / 7.0 / 8.3 / 13.2 / 12.8 / 22.2 us in a replayed graph
// (on the CUDA cores 9.2 / 8.1 / 10.9 / 15.1 / 15.9 / 23.6), two projections called one after the other, which overlap more, 5.4 / 6.6 /
// 8.6 / 11.4 / 11.8 / 18.5 (launch after launch: 6.5 / 7.6 / 9.3 / 13.8 / 13.4 / 22.8 and 8.5 / 8.0 / 9.2 / 12.2 / 12.7 / 19.5).  A row
// keeps the order of its sums by it, which differs between the two.
constexpr int kFusedDefaultRows = 1;
constexpr int kFusedMaxSlots = 12;
constexpr int kFusedItemRows = 16;  // gate/up rows per ring item of the eight-column kernel
constexpr int kFusedSmem = 227 * 1024 - 1040;              // one CTA per SM, beside what the kernels declare
constexpr int kFusedOnePairSmem = 223 * 512;               // two CTAs per SM
constexpr int kFusedMaxGrid = 256;
constexpr unsigned int kFusedPatienceNs = 100000;

enum FusedWaitCode : unsigned int {
    kWaitFusedFull = 0x201,
    kWaitFusedEmpty = 0x202,
    kWaitFusedMeeting = 0x203,       // reported by the self test alone: a CTA of an MLP that waits in vain leaves its rows
    kWaitFusedMeetingWrong = 0x2FF,  // ... whose meeting did not go as it should
};

// Where the CTAs of a launch meet.  Launches that may run at the same time have different slots (meeting_slots.h).  Every launch
// adds exactly gridDim.x to its count, so a count is always a multiple of the grid size between uses, and every flag down, but
// behind a launch that gave up (a copy that never landed); mt_device_status(reset) then zeroes them all.
struct __align__(64) FusedMeetingSlot {
    unsigned long long count;
    unsigned int left[kFusedMaxGrid / 32];  // down rows that their CTA has left to the last CTA of the launch, a bit per CTA
};
__device__ FusedMeetingSlot g_fused_meetings[kMeetingSlotsInAll];

struct FusedMeetingPlace {
    FusedMeetingSlot* slot;
    unsigned int patience_ns;
};

struct FusedMlpParams {
    CUtensorMap gate_map;      // gate_w / up_w as [I, H/8] uint32 tensors, boxes of 32 words x a tile's rows with the
    CUtensorMap up_map;        // 128-byte swizzle
    CUtensorMap down_map;      // down_w as [H, I/8], one-row kernel only
    const uint16_t* x;         // [1, H] bf16
    const uint32_t* gate_w;    // [I, H/8]
    const uint32_t* up_w;      // [I, H/8]
    const uint32_t* down_w;    // [H, I/8]
    const uint16_t* gate_s;    // [I, H/64]
    const uint16_t* gate_b;
    const uint16_t* up_s;
    const uint16_t* up_b;
    const uint16_t* down_s;    // [H, I/64]
    const uint16_t* down_b;
    const uint16_t* residual;  // [1, H] or null
    uint16_t* hidden;          // [1, I] bf16, written then read
    uint16_t* out;             // [1, H]
    FusedMeetingPlace meeting;
    int M, H, I;
};

__host__ __device__ inline int fused_round16(int v) { return (v + 15) & ~15; }

// Shared memory of the one-row kernel.
struct FusedOneLayout {
    int rows1_max, rows2_max;  // most rows any CTA owns in each projection
    int tile1, tile2;          // rows of a tile
    int chunks1, chunks2;      // 512-column units of a weight row
    int depth;                 // units in a warp's ring
    int tables1, tables2, scratch, bars, total;  // byte offsets; the rings come first
};

__host__ __device__ inline FusedOneLayout fused_one_layout(int M, int H, int I, int grid) {
    FusedOneLayout l;
    l.rows1_max = (I + grid - 1) / grid;
    l.rows2_max = (H + grid - 1) / grid;
    const int tiles1 = (l.rows1_max + 15) / 16, tiles2 = (l.rows2_max + 15) / 16;
    l.tile1 = (l.rows1_max + tiles1 - 1) / tiles1;
    l.tile2 = (l.rows2_max + tiles2 - 1) / tiles2;
    l.chunks1 = H / 512;
    l.chunks2 = I / 512;
    const int tables1 = 4 * l.rows1_max * (H >> 5), tables2 = 2 * l.rows2_max * (I >> 5);
    const int floats1 = l.rows1_max * 2 * l.chunks1 * M, floats2 = l.rows2_max * l.chunks2 * M;
    const int scratch = fused_round16(4 * (floats1 > floats2 ? floats1 : floats2));
    const int units = (tiles1 * 2 * l.chunks1 + kFusedOneWarps - 1) / kFusedOneWarps + (tiles2 * l.chunks2 + kFusedOneWarps - 1) / kFusedOneWarps;
    constexpr int kBars = 8 * (kFusedOneWarps * kFusedMaxSlots + 2) + 16;
    const int fixed = 1024 + tables1 + tables2 + scratch + kBars;
    const bool pair = kFusedOnePairSmem - fixed >= 2 * kFusedOneWarps * kOneRowItemBytes;
    const int left = (pair ? kFusedOnePairSmem : kFusedSmem) - fixed;
    l.depth = left / (kFusedOneWarps * kOneRowItemBytes);
    if (l.depth > units) l.depth = units;
    if (l.depth > kFusedMaxSlots) l.depth = kFusedMaxSlots;
    l.tables1 = l.depth * kFusedOneWarps * kOneRowItemBytes;
    l.tables2 = l.tables1 + tables1;
    l.scratch = l.tables2 + tables2;
    l.bars = l.scratch + scratch;
    l.total = l.bars + kBars;
    return l;
}

// Shared memory of the eight-column kernel.
struct FusedMlpLayout {
    int item_bytes, slots;     // ring geometry
    int down_rows;             // down rows per ring item
    int ring, scratch, bars, total;  // byte offsets
};

// Ring items (all the same size): gate|up item = 16 rows of gate, 16 rows of up and their four
// 16-row blocks of scales and biases (18*H bytes); down item = 32*H/I rows of down with their
// scales and biases.
__host__ __device__ inline FusedMlpLayout fused_mlp_layout(int H, int I) {
    FusedMlpLayout l;
    l.item_bytes = kFusedItemRows * (H + H / 8);  // rows x (H/2 gate + H/2 up) + rows x 4 x H/32
    int down = (2 * kFusedItemRows * H) / I;      // rows r with r * (I/2 + 2 * I/32) <= item_bytes
    if (down > 2 * kFusedItemRows) down = 2 * kFusedItemRows;
    if (down > 8) down -= down % 8;  // whole 8-row halves of a 16-row fragment
    l.down_rows = down;
    const int scratch_bytes = 4 * kFusedComputeWarps * 2 * 16 * 8;  // per-item partial tiles
    const int bars_bytes = 8 * (2 * kFusedMaxSlots) + 16;
    const int fixed = scratch_bytes + bars_bytes + 128;
    int slots = (kFusedSmem - fixed) / l.item_bytes;
    if (slots > kFusedMaxSlots) slots = kFusedMaxSlots;
    l.slots = slots;
    l.ring = 0;
    l.scratch = l.ring + slots * l.item_bytes;
    l.bars = l.scratch + scratch_bytes;
    l.total = l.bars + bars_bytes;
    return l;
}

// Barrier among the compute warps only (the producer warp keeps feeding the ring).
__device__ __forceinline__ void fused_compute_sync() {
    asm volatile("bar.sync 1, %0;" ::"r"(kFusedComputeThreads) : "memory");
}

// The producer warp of the eight-column kernel: streams the CTA's items through the ring.  Weights do
// not depend on the preceding kernel, so nothing here waits for it.  The gate|up rows of an item arrive as
// 128-byte-wide tensor-map boxes (32 words x 16 rows, 128-byte swizzle; layout [matrix][H/256 column
// blocks][16 rows][128 B]), which keeps the fragment loads free of bank conflicts.  A box is always 16
// rows: rows past the CTA's share (or past the tensor, zero-filled) are simply not used.  `first`: items before these, 0 or
// (other CTAs' down rows, which fit the ring) all of them read.
__device__ __forceinline__ void fused_producer(const FusedMlpParams& p, const FusedMlpLayout& lay, uint8_t* ring,
                                               uint64_t* full_bar, uint64_t* empty_bar, volatile int* abort_flag,
                                               int lane, int first, int row1, int n1, int row2, int n2) {
    const int H = p.H, I = p.I;
    const int items1 = (n1 + kFusedItemRows - 1) / kFusedItemRows;
    const int items2 = (n2 + lay.down_rows - 1) / lay.down_rows;
    const int rb1 = H >> 1, rb2 = I >> 1, sb1 = H >> 5, sb2 = I >> 5;
    const int slots = lay.slots;
    for (int it = 0; it < items1 + items2; ++it) {
        const int slot = (first + it) % slots, use = (first + it) / slots;
        if (use > 0 && first == 0 && !ptx::mbar_wait(&empty_bar[slot], (uint32_t)(use - 1) & 1u, abort_flag, kWaitFusedEmpty)) break;
        __syncwarp();
        uint8_t* dst = ring + (size_t)slot * lay.item_bytes;
        if (it < items1) {
            const int rows = min(kFusedItemRows, n1 - kFusedItemRows * it);
            const size_t r0 = (size_t)(row1 + kFusedItemRows * it);
            const int blocks = H >> 8;  // 256 columns = 128 packed bytes per box
            if (lane == 0)
                ptx::mbar_expect_tx(&full_bar[slot], (uint32_t)(2 * kFusedItemRows * rb1) + (uint32_t)rows * (uint32_t)(4 * sb1));
            __syncwarp();
            for (int box = lane; box < 2 * blocks; box += 32) {
                const int matrix = box / blocks, block = box - matrix * blocks;
                ptx::tma_load_2d(dst + (size_t)box * (kFusedItemRows * 128), matrix ? &p.up_map : &p.gate_map, block * 32,
                                 (int)r0, &full_bar[slot]);
            }
            if (lane >= 28) {
                const int which = lane - 28;
                const uint16_t* base = which == 0 ? p.gate_s : which == 1 ? p.gate_b : which == 2 ? p.up_s : p.up_b;
                ptx::bulk_load(dst + 2 * kFusedItemRows * rb1 + which * kFusedItemRows * sb1,
                               base + r0 * (size_t)(H >> 6), (uint32_t)rows * sb1, &full_bar[slot]);
            }
        } else {
            const int j = it - items1;
            const int rows = min(lay.down_rows, n2 - lay.down_rows * j);
            const size_t r0 = (size_t)(row2 + lay.down_rows * j);
            if (lane == 0) ptx::mbar_expect_tx(&full_bar[slot], (uint32_t)rows * (uint32_t)(rb2 + 2 * sb2));
            __syncwarp();
            if (lane == 0) {
                ptx::bulk_load(dst, p.down_w + r0 * (size_t)(I >> 3), (uint32_t)rows * rb2, &full_bar[slot]);
            } else if (lane < 3) {
                const uint16_t* base = lane == 1 ? p.down_s : p.down_b;
                ptx::bulk_load(dst + lay.down_rows * rb2 + (lane - 1) * lay.down_rows * sb2,
                               base + r0 * (size_t)(I >> 6), (uint32_t)rows * sb2, &full_bar[slot]);
            }
        }
    }
}

// How the CTAs of both kernels meet between the projections, in an ordinary launch (a cooperative one does not begin before the
// kernel in front has left the chip: 2048 / 8192, launch after launch, 16.2 us, so 13.0).  Nothing then says that all CTAs are on
// the chip together: beside another stream's kernel, or another such launch, some may not start before others have left.  So
// none waits for good: a CTA whose patience ends leaves its down rows to the last CTA to arrive, and makes room.
//
// The slot counts arrivals and, from bit 48, CTAs that have left their rows: one word, so the last arrival and a leaving CTA see one
// another in its order.  A flag is raised before its CTA is counted, and whoever lowers it has the rows and takes the CTA off the
// count again.
enum FusedMeeting : int { kMeetOpen, kMeetLast, kMeetLeft };  // kMeetLast: the last one, where some have left
constexpr unsigned long long kMeetOneLeft = 1ull << 48;

__device__ __forceinline__ int fused_meet(const FusedMeetingPlace& at, unsigned int grid, unsigned int cta) {
    unsigned long long* const count = &at.slot->count;
    // Release: the hidden activations of this CTA (ordered by the caller's barrier) are visible to whoever acquires the count.
    const unsigned long long before = ptx::atom_add_acq_rel_gpu_u64(count, 1ull), arrived = before % kMeetOneLeft;
    const unsigned long long target = (arrived / grid + 1ull) * grid;
    if (arrived + 1ull == target) return before >= kMeetOneLeft ? kMeetLast : kMeetOpen;
    const unsigned long long start = ptx::global_timer_ns();
    while (ptx::ld_acquire_gpu_u64(count) % kMeetOneLeft < target) {
        if (ptx::global_timer_ns() - start < at.patience_ns) continue;
        unsigned int* const flags = at.slot->left + (cta >> 5);
        const unsigned int mine = 1u << (cta & 31u);
        atomicOr(flags, mine);
        if (ptx::atom_add_acq_rel_gpu_u64(count, kMeetOneLeft) % kMeetOneLeft < target) return kMeetLeft;
        if (!(atomicAnd(flags, ~mine) & mine)) return kMeetLeft;  // the last CTA saw the flag on its way to another's
        ptx::atom_add_acq_rel_gpu_u64(count, 0ull - kMeetOneLeft);
        return kMeetOpen;
    }
    return kMeetOpen;
}

// Takes over the rows of `cta` if it has left them.
__device__ __forceinline__ void fused_take_over(const FusedMeetingPlace& at, unsigned int cta, int* taken, int* count) {
    const unsigned int its = 1u << (cta & 31u);
    if (!(atomicAnd(at.slot->left + (cta >> 5), ~its) & its)) return;
    taken[atomicAdd(count, 1)] = (int)cta;
    ptx::atom_add_acq_rel_gpu_u64(&at.slot->count, 0ull - kMeetOneLeft);
}

// Lane (g, t)'s activations of a 512-column unit: the B registers of one_row_products, and the sums of groups 2t and 2t + 1 in kOneRowUnit.
template <bool kFromL2>
__device__ __forceinline__ void fused_one_activations(const uint16_t* unit, int g, int t, uint32_t (&xr)[16], float2& sums) {
    const bool carries = (g & 1) == (t >> 1);  // whether column g belongs to this lane's half of the groups
    float total = 0.0f;
#pragma unroll
    for (int u = 0; u < 4; ++u) {
        const uint16_t* from = unit + g * 64 + (t & 1) * 32 + u * 8;
        uint4 v = make_uint4(0u, 0u, 0u, 0u);
        if (carries) v = kFromL2 ? ptx::ld_global_l2_u4(from) : ptx::ld_global_dependent_u4(from);
        total += ((bf16_lo(v.x) + bf16_hi(v.x)) + (bf16_lo(v.y) + bf16_hi(v.y))) + ((bf16_lo(v.z) + bf16_hi(v.z)) + (bf16_lo(v.w) + bf16_hi(v.w)));
        xr[4 * u] = __byte_perm(v.x, v.z, 0x5410);
        xr[4 * u + 1] = __byte_perm(v.x, v.z, 0x7632);
        xr[4 * u + 2] = __byte_perm(v.y, v.w, 0x5410);
        xr[4 * u + 3] = __byte_perm(v.y, v.w, 0x7632);
    }
    total = kOneRowUnit * (total + __shfl_xor_sync(0xFFFFFFFFu, total, 1));
    sums.x = __shfl_sync(0xFFFFFFFFu, total, 8 * t);      // group 2t: lanes (2t, 0) and (2t, 1)
    sums.y = __shfl_sync(0xFFFFFFFFu, total, 8 * t + 6);  // group 2t + 1: lanes (2t + 1, 2) and (2t + 1, 3)
}

__global__ void __launch_bounds__(kFusedOneThreads, 2)
affine_mlp_fused_kernel(const __grid_constant__ FusedMlpParams p) {
    extern __shared__ uint8_t fused_smem_raw[];
    // 1024-byte alignment: the swizzle pattern of the tensor-map boxes repeats every 1024 bytes.
    uint8_t* smem = fused_smem_raw + ((1024u - (ptx::smem_u32(fused_smem_raw) & 1023u)) & 1023u);  // stays a shared-memory address
    const int grid = gridDim.x, cta = blockIdx.x;
    const int M = p.M, H = p.H, I = p.I;
    const FusedOneLayout lay = fused_one_layout(M, H, I, grid);
    const int warp = __shfl_sync(0xFFFFFFFFu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    const int depth = lay.depth;
    uint8_t* ring = smem + warp * depth * kOneRowItemBytes;
    float* scratch = reinterpret_cast<float*>(smem + lay.scratch);
    uint64_t* unit_full = reinterpret_cast<uint64_t*>(smem + lay.bars) + warp * depth;
    uint64_t* table_full = reinterpret_cast<uint64_t*>(smem + lay.bars) + kFusedOneWarps * kFusedMaxSlots;
    volatile int* abort_flag = reinterpret_cast<volatile int*>(table_full + 2);
    __shared__ int meeting, left_count, left_ctas[kFusedMaxGrid];

    const int row1 = (int)((unsigned)I * (unsigned)cta / (unsigned)grid);
    const int n1 = (int)((unsigned)I * (unsigned)(cta + 1) / (unsigned)grid) - row1;
    int row2, n2, units2;
    // Units in the order (tile, matrix, chunk); where the chunks of a tile divide the warps a warp's chunk never changes (always in
    // gate|up).
    const int per_tile1 = 2 * lay.chunks1, units1 = (n1 + lay.tile1 - 1) / lay.tile1 * per_tile1;
    const int per_tile2 = lay.chunks2;
    auto down_rows_of = [&](int owner) {
        row2 = (int)((unsigned)H * (unsigned)owner / (unsigned)grid);
        n2 = (int)((unsigned)H * (unsigned)(owner + 1) / (unsigned)grid) - row2;
        units2 = (n2 + lay.tile2 - 1) / lay.tile2 * per_tile2;
    };
    down_rows_of(cta);
    const int chunk1 = warp & (lay.chunks1 - 1);

    if (threadIdx.x == 0) {
        for (int i = 0; i < kFusedOneWarps * depth; ++i) ptx::mbar_init(reinterpret_cast<uint64_t*>(smem + lay.bars) + i, 1);
        ptx::mbar_init(&table_full[0], 1);
        ptx::mbar_init(&table_full[1], 1);
        *abort_flag = 0;
        left_count = 0;
        ptx::mbar_fence_init();
    }
    __syncthreads();
    ptx::griddep_launch_dependents();

    // ---- the copies of this warp's units: those of gate|up, then those of down
    int copy_unit = warp;
    bool copy_down = false;
    auto copy_next = [&](int slot) {
        if (!copy_down && copy_unit >= units1) {
            copy_down = true;
            copy_unit = warp;
        }
        if (copy_down && copy_unit >= units2) return;
        if (ptx::elect_one()) {
            uint8_t* to = ring + slot * kOneRowItemBytes;
            const int per_tile = copy_down ? per_tile2 : per_tile1, tile = copy_unit / per_tile;
            const int rows = copy_down ? lay.tile2 : lay.tile1, at = (copy_down ? row2 : row1) + tile * rows;
            const bool up = !copy_down && copy_unit - tile * per_tile >= lay.chunks1;
            const CUtensorMap* map = copy_down ? &p.down_map : up ? &p.up_map : &p.gate_map;
            ptx::mbar_expect_tx(&unit_full[slot], 256u * (uint32_t)rows);
#pragma unroll
            for (int i = 0; i < 2; ++i)  // rows past the CTA's share are not used, past the matrix filled with zeros
                ptx::tma_load_2d(to + i * 2048, map, (copy_down ? copy_unit & (lay.chunks2 - 1) : chunk1) * 64 + i * 32, at, &unit_full[slot]);
        }
        __syncwarp();
        copy_unit += kFusedOneWarps;
    };
    copy_next(0);
    if (warp == 0 && ptx::elect_one()) {  // the tables of all rows of this CTA
        const uint32_t bytes1 = (uint32_t)n1 * (uint32_t)(H >> 5);
        const uint16_t* const tables1[4] = {p.gate_s, p.gate_b, p.up_s, p.up_b};
        ptx::mbar_expect_tx(&table_full[0], 4u * bytes1);
#pragma unroll
        for (int i = 0; i < 4; ++i)
            ptx::bulk_load(smem + lay.tables1 + i * lay.rows1_max * (H >> 5), tables1[i] + (size_t)row1 * (H >> 6), bytes1, &table_full[0]);
    }
    __syncwarp();
    auto copy_down_tables = [&] {
        if (warp == 0 && ptx::elect_one()) {
            const uint32_t bytes = (uint32_t)n2 * (uint32_t)(I >> 5);
            const uint16_t* const from[2] = {p.down_s, p.down_b};
            ptx::mbar_expect_tx(&table_full[1], 2u * bytes);
#pragma unroll
            for (int i = 0; i < 2; ++i)
                ptx::bulk_load(smem + lay.tables2 + i * lay.rows2_max * (I >> 5), from[i] + (size_t)row2 * (I >> 6), bytes, &table_full[1]);
        }
        __syncwarp();
    };
    copy_down_tables();
    for (int slot = 1; slot < depth; ++slot) copy_next(slot);

    ptx::griddep_wait();  // the activations and the residual are the preceding kernel's output
    float residual_value;  // fetched now, used at the very end
    auto fetch_residual = [&] {
        residual_value = 0.0f;
        if ((int)threadIdx.x < n2 * M && p.residual) {
            const int row = threadIdx.x / M, m = threadIdx.x - row * M;
            residual_value = bf16_bits_to_f32(ptx::ld_global_dependent_u16(p.residual + (size_t)m * H + row2 + row));
        }
    };
    fetch_residual();
    const int tile_row = one_row_tile_row(g);
    bool alive = true;
    int slot = 0;
    uint32_t phase = 0, down_tables_phase = 0;  // phase: a bit per slot
    // Sums of this warp's units, to scratch[((row * matrices + matrix) * chunks + chunk) * M + m].
    auto project = [&](auto down) {
        constexpr bool kDown = decltype(down)::value;
        const int units = kDown ? units2 : units1, per_tile = kDown ? per_tile2 : per_tile1, tile_rows = kDown ? lay.tile2 : lay.tile1;
        const int n = kDown ? n2 : n1, chunks = kDown ? lay.chunks2 : lay.chunks1, chunk0 = kDown ? warp & (lay.chunks2 - 1) : chunk1;
        const int width = kDown ? I : H, groups = width >> 6;
        const int table = (kDown ? lay.rows2_max : lay.rows1_max) * (width >> 5);
        const uint8_t* tables = smem + (kDown ? lay.tables2 : lay.tables1);
        const uint16_t* x = kDown ? p.hidden : p.x;
        if (warp >= units) return;
        uint32_t xr[16];
        float2 xs;
        fused_one_activations<kDown>(x + chunk0 * 512, g, t, xr, xs);
        if (alive) alive = __all_sync(0xFFFFFFFFu, ptx::mbar_wait(&table_full[kDown], kDown ? down_tables_phase : 0u, abort_flag, kWaitFusedFull));
        for (int unit = warp; unit < units; unit += kFusedOneWarps) {
            if (alive) alive = __all_sync(0xFFFFFFFFu, ptx::mbar_wait(&unit_full[slot], (phase >> slot) & 1u, abort_flag, kWaitFusedFull));
            if (!alive) return;
            phase ^= 1u << slot;
            uint32_t row[4][4], row8[4][4];
            one_row_words(ring + slot * kOneRowItemBytes, tile_row, t, row, row8);
            ptx::fence_proxy_async_smem();  // the slot is filled again
            __syncwarp();
            copy_next(slot);
            if (++slot == depth) slot = 0;
            const int chunk = kDown ? unit & (lay.chunks2 - 1) : chunk0;
            const int tile = unit / per_tile, matrix = !kDown && unit - tile * per_tile >= lay.chunks1 ? 1 : 0;
            const int first = tile * tile_rows, last = min(first + tile_rows, n) - 1;
            const uint8_t* scales = tables + 2 * matrix * table;
            uint32_t scale[2], bias[2];  // of groups 2t and 2t + 1 of this lane's rows
#pragma unroll
            for (int r = 0; r < 2; ++r) {
                const int at = (min(first + tile_row + 8 * r, last) * groups + chunk * kOneRowItemGroups + 2 * t) * 2;
                scale[r] = *reinterpret_cast<const uint32_t*>(scales + at);
                bias[r] = *reinterpret_cast<const uint32_t*>(scales + table + at);
            }
            for (int m = 0; m < M; ++m) {
                if (M > 1 || (kDown && lay.chunks2 > kFusedOneWarps && unit != warp)) fused_one_activations<kDown>(x + (size_t)m * width + chunk * 512, g, t, xr, xs);
                float own[4], total[2];
                one_row_products(row, row8, xr, t, own);
#pragma unroll
                for (int r = 0; r < 2; ++r) {
                    const float s0 = bf16_lo(scale[r]), s1 = bf16_hi(scale[r]);
                    const float b0 = fmaf(8.0f, s0, bf16_lo(bias[r])), b1 = fmaf(8.0f, s1, bf16_hi(bias[r]));  // the products are of (q - 8) / 64, xs is X / 64
                    total[r] = fmaf(s0, own[2 * r], b0 * xs.x);
                    total[r] = fmaf(s1, own[2 * r + 1], fmaf(b1, xs.y, total[r]));
                    total[r] += __shfl_xor_sync(0xFFFFFFFFu, total[r], 1);
                    total[r] += __shfl_xor_sync(0xFFFFFFFFu, total[r], 2);
                }
                const int mine = first + tile_row + 8 * (t & 1);
                if (t < 2 && mine <= last)
                    scratch[((mine * (kDown ? 1 : 2) + matrix) * chunks + chunk) * M + m] = (t == 0 ? total[0] : total[1]) / kOneRowUnit;
            }
        }
    };
    project(std::false_type{});
    __syncthreads();
    for (int idx = threadIdx.x; idx < n1 * M; idx += kFusedOneThreads) {
        const int row = idx / M, m = idx - row * M;
        float gate = 0.0f, up = 0.0f;
        for (int c = 0; c < lay.chunks1; ++c) {
            gate += scratch[((2 * row + 0) * lay.chunks1 + c) * M + m];
            up += scratch[((2 * row + 1) * lay.chunks1 + c) * M + m];
        }
        p.hidden[(size_t)m * I + row1 + row] = f32_to_bf16_bits(swiglu_f32(gate, up));
    }
    __syncthreads();
    if (threadIdx.x == 0) meeting = fused_meet(p.meeting, (unsigned)grid, (unsigned)cta);
    __syncthreads();
    const int met = meeting;
    for (int next = 0;; ++next) {
        project(std::true_type{});  // of a CTA that has left its rows, too: its copies have then landed
        __syncthreads();
        if (met != kMeetLeft && (int)threadIdx.x < n2 * M) {
            const int row = threadIdx.x / M, m = threadIdx.x - row * M;
            float v = 0.0f;
            for (int c = 0; c < lay.chunks2; ++c) v += scratch[(row * lay.chunks2 + c) * M + m];
            p.out[(size_t)m * H + row2 + row] = f32_to_bf16_bits(v + residual_value);
        }
        if (met != kMeetLast) break;
        if (next == 0 && (int)threadIdx.x < grid) fused_take_over(p.meeting, threadIdx.x, left_ctas, &left_count);
        ptx::fence_proxy_async_smem();  // the tables are filled again
        __syncthreads();
        if (next == left_count || *abort_flag) break;
        down_rows_of(left_ctas[next]);
        copy_unit = warp;
        copy_down_tables();
        for (int i = 0; i < depth; ++i) copy_next(slot + i < depth ? slot + i : slot + i - depth);
        fetch_residual();
        down_tables_phase ^= 1u;
    }
    if (*abort_flag) ptx::drain_copies();
}

// ===================================================================================================
// Eight-column kernel for two to eight activation rows.
//
// The multiply runs on mma.sync (m16n8k16, bf16 in, fp32 out): the A fragment is exactly
// what the nibble unpack produces -- bf16 pairs (128+q_i, 128+q_{i+4}), 7 integer instructions per
// packed word -- and up to eight activation rows ride in the B fragment for free.  Four MMAs cover one
// quantisation group (64 k) of 16 weight rows; the group's partial sums P are folded as
// acc += s * P + (b - 128 s) * X, X = the group's activation sum, so weights stay exact.  The four MMAs of a group are a dependent chain,
// so four (block, group) pairs are issued round-robin; with one chain at a time the kernel took 25 us.
// The fragment loads are 64 bits per lane from four weight rows at a time; in a dense row layout those
// rows share their banks (4-way conflicts, 1.5 M extra wavefronts per launch), so the gate|up rows arrive
// as 128-byte-swizzled tensor-map boxes and fragment row g is given weight row 2 (g % 4) + g / 4, which
// makes the four rows' swizzles differ; scales and biases are read four groups per load (their rows lie
// 64 or 256 bytes apart, again in the same banks).  Steps of its making at 2048 / 8192, eight rows, in a cooperative launch: one
// chain 25.6 us, four 22.5, swizzled boxes 20.1, wide table loads 19.5; in the ordinary launch of now 18.5 in a
// replayed graph and 18.3 called from Python (20.5 before).  Why two to eight rows take it: see mt_affine_mlp.
//
// A producer warp feeds one ring; the CTAs meet as above.  The K range is cut into one slice per compute warp; every
// warp walks all rows of an item for its slice; the warps' partial 16 x 8 tiles meet in shared memory
// and are added in warp order.  Activation fragments hold element pairs in the order the unpack emits
// them: (e0,e4), (e1,e5), (e2,e6), (e3,e7).

constexpr int kFusedMmaMaxRows = 8;
constexpr int kFusedMmaMaxGroups1 = 4;  // quantisation groups of H per warp that fit in registers

__device__ __forceinline__ uint4 permute_for_fragment(uint4 v) {
    uint4 o;
    o.x = __byte_perm(v.x, v.z, 0x5410);
    o.y = __byte_perm(v.x, v.z, 0x7632);
    o.z = __byte_perm(v.y, v.w, 0x5410);
    o.w = __byte_perm(v.y, v.w, 0x7632);
    return o;
}

// Lane (g, t) loads column g's 16 activations k = 64 group + 16 t .. +15 as two fragment registers
// sets, and returns the group's sums of columns 2t and 2t+1 (x0, x1) gathered by shuffles.
template <bool kFromL2>
__device__ __forceinline__ void load_group_fragments(const uint16_t* column, bool active, int group, int t, uint4& bx0,
                                                     uint4& bx1, float& x0, float& x1) {
    uint4 v0 = make_uint4(0, 0, 0, 0), v1 = make_uint4(0, 0, 0, 0);
    if (active) {
        const uint16_t* from = column + group * 64 + t * 16;
        v0 = kFromL2 ? ptx::ld_global_l2_u4(from) : ptx::ld_global_dependent_u4(from);
        v1 = kFromL2 ? ptx::ld_global_l2_u4(from + 8) : ptx::ld_global_dependent_u4(from + 8);
    }
    bx0 = permute_for_fragment(v0);
    bx1 = permute_for_fragment(v1);
    const uint32_t words[8] = {v0.x, v0.y, v0.z, v0.w, v1.x, v1.y, v1.z, v1.w};
    float partial = 0.0f;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        partial += bf16_lo(words[i]);
        partial += bf16_hi(words[i]);
    }
    partial += __shfl_xor_sync(0xFFFFFFFFu, partial, 1);
    partial += __shfl_xor_sync(0xFFFFFFFFu, partial, 2);  // every lane of fragment row g holds column g's sum
    x0 = __shfl_sync(0xFFFFFFFFu, partial, 8 * t);        // lane 4 * (2t)
    x1 = __shfl_sync(0xFFFFFFFFu, partial, 8 * t + 4);    // lane 4 * (2t + 1)
}

// kN independent (16-row block, quantisation group) pairs at once: rows g (lower) and g+8 (upper) of
// each fragment.  The four MMAs of a pair form a dependent chain (they accumulate one group's partial
// sums), so the pairs' MMAs are issued round-robin to keep the tensor pipe fed.
// Four consecutive bf16 table entries (scales or biases of groups group..group+3 of one row) as one
// 64-bit load when they are 8-byte aligned, else entry by entry; entries past `count` are not read.
__device__ __forceinline__ uint2 load_four_entries(const uint8_t* row, int group, int count) {
    if (((group & 3) == 0) && count >= 4) return *reinterpret_cast<const uint2*>(row + group * 2);
    uint32_t e[4] = {0, 0, 0, 0};
#pragma unroll
    for (int i = 0; i < 4; ++i)
        if (i < count) e[i] = *reinterpret_cast<const uint16_t*>(row + (group + i) * 2);
    return make_uint2(e[0] | (e[1] << 16), e[2] | (e[3] << 16));
}
__device__ __forceinline__ uint32_t entry_of(uint2 four, int i) {
    const uint32_t word = i < 2 ? four.x : four.y;
    return (i & 1) ? word >> 16 : word & 0xFFFFu;
}

struct MmaOperand {
    const uint8_t* lower;   // this lane's 8 packed bytes of row g for the group
    const uint8_t* upper;   // ... of row g+8 (ignored without kUpper)
    uint32_t scale_lo, bias_lo, scale_hi, bias_hi;  // bf16 bits
};

template <int kN, bool kUpper>
__device__ __forceinline__ void mma_groups(const MmaOperand (&op)[kN], const uint4 (&bx0)[kN], const uint4 (&bx1)[kN],
                                           const float (&x0)[kN], const float (&x1)[kN], float* const (&acc)[kN]) {
    uint32_t lo[kN][8], hi[kN][8];
#pragma unroll
    for (int i = 0; i < kN; ++i) {
        const uint2 l = *reinterpret_cast<const uint2*>(op[i].lower);
        unpack_word_offset128(l.x, &lo[i][0]);
        unpack_word_offset128(l.y, &lo[i][4]);
        if constexpr (kUpper) {
            const uint2 h = *reinterpret_cast<const uint2*>(op[i].upper);
            unpack_word_offset128(h.x, &hi[i][0]);
            unpack_word_offset128(h.y, &hi[i][4]);
        } else {
#pragma unroll
            for (int k = 0; k < 8; ++k) hi[i][k] = 0u;
        }
    }
    float d[kN][4];
#pragma unroll
    for (int i = 0; i < kN; ++i) d[i][0] = d[i][1] = d[i][2] = d[i][3] = 0.0f;
#pragma unroll
    for (int i = 0; i < kN; ++i) ptx::mma_bf16_m16n8k16(d[i], lo[i][0], hi[i][0], lo[i][1], hi[i][1], bx0[i].x, bx0[i].y);
#pragma unroll
    for (int i = 0; i < kN; ++i) ptx::mma_bf16_m16n8k16(d[i], lo[i][2], hi[i][2], lo[i][3], hi[i][3], bx0[i].z, bx0[i].w);
#pragma unroll
    for (int i = 0; i < kN; ++i) ptx::mma_bf16_m16n8k16(d[i], lo[i][4], hi[i][4], lo[i][5], hi[i][5], bx1[i].x, bx1[i].y);
#pragma unroll
    for (int i = 0; i < kN; ++i) ptx::mma_bf16_m16n8k16(d[i], lo[i][6], hi[i][6], lo[i][7], hi[i][7], bx1[i].z, bx1[i].w);
#pragma unroll
    for (int i = 0; i < kN; ++i) {
        const float s_lo = bf16_bits_to_f32(op[i].scale_lo);
        const float o_lo = fmaf(-128.0f, s_lo, bf16_bits_to_f32(op[i].bias_lo));  // undoes the 128 in 128+q
        acc[i][0] = fmaf(s_lo, d[i][0], fmaf(o_lo, x0[i], acc[i][0]));
        acc[i][1] = fmaf(s_lo, d[i][1], fmaf(o_lo, x1[i], acc[i][1]));
        if constexpr (kUpper) {
            const float s_hi = bf16_bits_to_f32(op[i].scale_hi);
            const float o_hi = fmaf(-128.0f, s_hi, bf16_bits_to_f32(op[i].bias_hi));
            acc[i][2] = fmaf(s_hi, d[i][2], fmaf(o_hi, x0[i], acc[i][2]));
            acc[i][3] = fmaf(s_hi, d[i][3], fmaf(o_hi, x1[i], acc[i][3]));
        }
    }
}

__global__ void __launch_bounds__(kFusedThreads, 1)
affine_mlp_fused_mma_kernel(const __grid_constant__ FusedMlpParams p) {
    extern __shared__ uint8_t fused_smem_raw[];
    // 1024-byte alignment: the swizzle pattern of the tensor-map boxes repeats every 1024 bytes.
    uint8_t* smem = fused_smem_raw + ((1024u - (ptx::smem_u32(fused_smem_raw) & 1023u)) & 1023u);  // stays a shared-memory address
    const int grid = gridDim.x, cta = blockIdx.x;
    const int M = p.M, H = p.H, I = p.I;
    const FusedMlpLayout lay = fused_mlp_layout(H, I);
    uint8_t* ring = smem + lay.ring;
    float* scratch = reinterpret_cast<float*>(smem + lay.scratch);
    uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + lay.bars);
    uint64_t* empty_bar = full_bar + kFusedMaxSlots;
    volatile int* abort_flag = reinterpret_cast<volatile int*>(empty_bar + kFusedMaxSlots);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int g = lane >> 2, t = lane & 3;

    const int row1 = (int)((unsigned)I * (unsigned)cta / (unsigned)grid);
    const int n1 = (int)((unsigned)I * (unsigned)(cta + 1) / (unsigned)grid) - row1;
    int row2, n2, items2;
    auto down_rows_of = [&](int owner) {
        row2 = (int)((unsigned)H * (unsigned)owner / (unsigned)grid);
        n2 = (int)((unsigned)H * (unsigned)(owner + 1) / (unsigned)grid) - row2;
        items2 = (n2 + lay.down_rows - 1) / lay.down_rows;
    };
    down_rows_of(cta);
    const int items1 = (n1 + kFusedItemRows - 1) / kFusedItemRows;
    const int own_items = items1 + items2;
    int first_down = items1;  // items before the present down rows
    const int rb1 = H >> 1, rb2 = I >> 1, sb1 = H >> 5, sb2 = I >> 5;
    const int slots = lay.slots;

    __shared__ int meeting, left_count, left_ctas[kFusedMaxGrid], next_owner[2];
    if (threadIdx.x == 0) {
        left_count = 0;
        for (int i = 0; i < kFusedMaxSlots; ++i) {
            ptx::mbar_init(&full_bar[i], 1);
            ptx::mbar_init(&empty_bar[i], kFusedComputeWarps);
        }
        *abort_flag = 0;
        ptx::mbar_fence_init();
    }
    __syncthreads();
    ptx::griddep_launch_dependents();
    if (warp == kFusedComputeWarps) {
        if (lane == 0) {
            ptx::prefetch_tensor_map(&p.gate_map);
            ptx::prefetch_tensor_map(&p.up_map);
        }
        fused_producer(p, lay, ring, full_bar, empty_bar, abort_flag, lane, 0, row1, n1, row2, n2);
        for (int next = 0;; ++next) {  // down rows that others have left
            ptx::named_barrier_sync(2, kFusedThreads);
            const int owner = next_owner[next & 1];
            if (owner < 0) return;
            first_down += items2;
            down_rows_of(owner);
            fused_producer(p, lay, ring, full_bar, empty_bar, abort_flag, lane, first_down, 0, 0, row2, n2);
        }
    }

    // ---------------------------------------------------------------------- compute warps
    ptx::griddep_wait();  // the activations and the residual are the preceding kernel's output
    float residual_value;
    auto fetch_residual = [&] {
        residual_value = 0.0f;
        if ((int)threadIdx.x < n2 * M && p.residual) {
            const int row = threadIdx.x / M, m = threadIdx.x - row * M;
            residual_value = bf16_bits_to_f32(ptx::ld_global_dependent_u16(p.residual + (size_t)m * H + row2 + row));
        }
    };
    fetch_residual();
    const bool active = g < M;  // fragment column g carries activation row g
    bool alive = true;
    {
        // ------------------------------------------------------------------ gate | up
        const int groups = (H >> 6) / kFusedComputeWarps;  // quantisation groups in this warp's K slice (<= 4)
        const int group0 = warp * groups;
        // Fragment row g carries weight row 2 (g % 4) + g / 4 of each 8-row half: the four rows a half-warp
        // loads at once then differ in their swizzle by 0, 2, 4, 6 and hit disjoint banks.
        const int wrow = ((g & 3) << 1) | (g >> 2);
        uint4 bx0[kFusedMmaMaxGroups1], bx1[kFusedMmaMaxGroups1];
        float x0[kFusedMmaMaxGroups1], x1[kFusedMmaMaxGroups1];
#pragma unroll
        for (int gi = 0; gi < kFusedMmaMaxGroups1; ++gi)
            if (gi < groups) load_group_fragments<false>(p.x + (size_t)(active ? g : 0) * H, active, group0 + gi, t, bx0[gi], bx1[gi], x0[gi], x1[gi]);
        for (int it = 0; it < items1; ++it) {
            const int slot = it % slots, use = it / slots;
            if (alive && !ptx::mbar_wait(&full_bar[slot], (uint32_t)use & 1u, abort_flag, kWaitFusedFull)) alive = false;
            alive = __all_sync(0xFFFFFFFFu, alive);  // the MMAs and shuffles below need the whole warp or none of it
            const uint8_t* item = ring + (size_t)slot * lay.item_bytes;
            const uint8_t* tables = item + 2 * kFusedItemRows * rb1;
            const int rows_here = min(kFusedItemRows, n1 - kFusedItemRows * it);
            const bool upper = rows_here > 8;
            float acc[2][4] = {{0.0f, 0.0f, 0.0f, 0.0f}, {0.0f, 0.0f, 0.0f, 0.0f}};
            if (alive) {
                // This warp's scales and biases of the item: rows wrow and wrow + 8, gate and up, four groups each.
                uint2 sc4[2][2], bi4[2][2];  // [matrix][lower / upper]
#pragma unroll
                for (int matrix = 0; matrix < 2; ++matrix)
#pragma unroll
                    for (int half = 0; half < 2; ++half) {
                        const int row = wrow + 8 * half;
                        const bool present = half == 0 || upper;
                        sc4[matrix][half] = present ? load_four_entries(tables + ((2 * matrix) * kFusedItemRows + row) * sb1, group0, groups)
                                                    : make_uint2(0, 0);
                        bi4[matrix][half] = present ? load_four_entries(tables + ((2 * matrix + 1) * kFusedItemRows + row) * sb1, group0, groups)
                                                    : make_uint2(0, 0);
                    }
                // Two groups x (gate, up) = four independent MMA chains per step.  A second group past
                // the slice's end repeats the first one into a discarded accumulator.
#pragma unroll
                for (int gi = 0; gi < kFusedMmaMaxGroups1; gi += 2) {
                    if (gi < groups) {
                        const bool second = gi + 1 < groups;
                        float discard[4];
                        MmaOperand op[4];
                        uint4 fx0[4], fx1[4];
                        float fs0[4], fs1[4];
                        float* into[4];
#pragma unroll
                        for (int c = 0; c < 4; ++c) {
                            const int matrix = c & 1, which = (c >> 1) && second ? gi + 1 : gi;
                            const int group = group0 + which;
                            // Box (matrix, group / 4), row `wrow`, 16-byte chunk (group % 4) * 2 + t / 2 XOR-swizzled
                            // by the row; rows wrow and wrow + 8 share the swizzle.
                            const int chunk = (((group & 3) << 1) | (t >> 1)) ^ (wrow & 7);
                            op[c].lower = item + (size_t)((matrix * (H >> 8) + (group >> 2)) * kFusedItemRows + wrow) * 128 +
                                          (chunk << 4) + (t & 1) * 8;
                            op[c].upper = op[c].lower + 8 * 128;
                            op[c].scale_lo = entry_of(sc4[matrix][0], which);
                            op[c].bias_lo = entry_of(bi4[matrix][0], which);
                            op[c].scale_hi = entry_of(sc4[matrix][1], which);
                            op[c].bias_hi = entry_of(bi4[matrix][1], which);
                            fx0[c] = (c >> 1) && second ? bx0[(gi + 1) % kFusedMmaMaxGroups1] : bx0[gi];
                            fx1[c] = (c >> 1) && second ? bx1[(gi + 1) % kFusedMmaMaxGroups1] : bx1[gi];
                            fs0[c] = (c >> 1) && second ? x0[(gi + 1) % kFusedMmaMaxGroups1] : x0[gi];
                            fs1[c] = (c >> 1) && second ? x1[(gi + 1) % kFusedMmaMaxGroups1] : x1[gi];
                            into[c] = (c >> 1) && !second ? discard : acc[matrix];
                        }
                        // The two chains of one matrix add into the same accumulators: fold the second
                        // group's pair after the first by giving it its own accumulators.
                        float later[2][4] = {{0.0f, 0.0f, 0.0f, 0.0f}, {0.0f, 0.0f, 0.0f, 0.0f}};
                        if (second) { into[2] = later[0]; into[3] = later[1]; }
                        if (upper) mma_groups<4, true>(op, fx0, fx1, fs0, fs1, into);
                        else mma_groups<4, false>(op, fx0, fx1, fs0, fs1, into);
                        if (second) {
#pragma unroll
                            for (int k = 0; k < 4; ++k) {
                                acc[0][k] += later[0][k];
                                acc[1][k] += later[1][k];
                            }
                        }
                    }
                }
            }
            if (it + slots < own_items) {
                ptx::fence_proxy_async_smem();
                __syncwarp();
                if (lane == 0) ptx::mbar_arrive(&empty_bar[slot]);
            }
            // scratch[((warp * 2 + matrix) * 16 + row) * 8 + column]
#pragma unroll
            for (int matrix = 0; matrix < 2; ++matrix) {
                float* tile = scratch + (size_t)((warp * 2 + matrix) * 16) * 8;
                *reinterpret_cast<float2*>(tile + wrow * 8 + 2 * t) = make_float2(acc[matrix][0], acc[matrix][1]);
                *reinterpret_cast<float2*>(tile + (wrow + 8) * 8 + 2 * t) = make_float2(acc[matrix][2], acc[matrix][3]);
            }
            fused_compute_sync();
            for (int idx = threadIdx.x; idx < rows_here * M; idx += kFusedComputeThreads) {
                const int row = idx / M, m = idx - row * M;
                float gate = 0.0f, up = 0.0f;
                for (int w = 0; w < kFusedComputeWarps; ++w) {
                    gate += scratch[((w * 2 + 0) * 16 + row) * 8 + m];
                    up += scratch[((w * 2 + 1) * 16 + row) * 8 + m];
                }
                p.hidden[(size_t)m * I + row1 + kFusedItemRows * it + row] = f32_to_bf16_bits(swiglu_f32(gate, up));
            }
            fused_compute_sync();
        }
    }
    fused_compute_sync();
    if (threadIdx.x == 0) meeting = fused_meet(p.meeting, (unsigned)grid, (unsigned)cta);
    fused_compute_sync();
    const int met = meeting;
    for (int next = 0;; ++next) {
        // ------------------------------------------------------------------ down
        const int groups = (I >> 6) / kFusedComputeWarps;
        const int group0 = warp * groups;
        const uint16_t* column = p.hidden + (size_t)(active ? g : 0) * I;
        const int tiles = (n2 + 15) >> 4;
        int released = 0;  // down items handed back to the producer so far
        for (int tile = 0; tile < tiles; ++tile) {
            // Rows 16 tile + g (lower) and 16 tile + 8 + g (upper) of this CTA's down rows, wherever
            // their items sit in the ring.
            const int r_lo = 16 * tile, r_hi = 16 * tile + 8;
            const bool upper = r_hi < n2;
            const int j_lo = r_lo / lay.down_rows, j_hi = upper ? r_hi / lay.down_rows : j_lo;
            for (int j = j_lo; j <= j_hi; ++j) {
                const int it = first_down + j;
                if (alive && !ptx::mbar_wait(&full_bar[it % slots], (uint32_t)(it / slots) & 1u, abort_flag, kWaitFusedFull))
                    alive = false;
            }
            alive = __all_sync(0xFFFFFFFFu, alive);
            const uint8_t* item_lo = ring + (size_t)((first_down + j_lo) % slots) * lay.item_bytes;
            const uint8_t* item_hi = ring + (size_t)((first_down + j_hi) % slots) * lay.item_bytes;
            const int local_lo = r_lo - j_lo * lay.down_rows + g, local_hi = r_hi - j_hi * lay.down_rows + g;
            const uint8_t* lower = item_lo + local_lo * rb2 + t * 8;
            const uint8_t* upper_row = item_hi + local_hi * rb2 + t * 8;
            const uint8_t* sc_lo = item_lo + lay.down_rows * rb2 + local_lo * sb2;
            const uint8_t* sc_hi = item_hi + lay.down_rows * rb2 + local_hi * sb2;
            const int table = lay.down_rows * sb2;  // biases follow the scales
            float acc[4] = {0.0f, 0.0f, 0.0f, 0.0f};
            if (alive) {
                // Four groups = four independent MMA chains per step; their activation fragments come
                // from L2 one step ahead.  Chains past the slice's end repeat the step's first group
                // into a discarded accumulator.
                uint4 bx0[4], bx1[4], nx0[4], nx1[4];
                float x0[4], x1[4], y0[4], y1[4];
#pragma unroll
                for (int c = 0; c < 4; ++c)
                    load_group_fragments<true>(column, active, group0 + (c < groups ? c : 0), t, bx0[c], bx1[c], x0[c], x1[c]);
                for (int gi = 0; gi < groups; gi += 4) {
                    if (gi + 4 < groups) {
#pragma unroll
                        for (int c = 0; c < 4; ++c)
                            load_group_fragments<true>(column, active, group0 + (gi + 4 + c < groups ? gi + 4 + c : gi + 4), t,
                                                       nx0[c], nx1[c], y0[c], y1[c]);
                    }
                    MmaOperand op[4];
                    float part[4][4];
                    float* into[4];
                    const int step_groups = min(4, groups - gi);
                    const uint2 s_lo4 = load_four_entries(sc_lo, group0 + gi, step_groups);
                    const uint2 b_lo4 = load_four_entries(sc_lo + table, group0 + gi, step_groups);
                    const uint2 s_hi4 = upper ? load_four_entries(sc_hi, group0 + gi, step_groups) : make_uint2(0, 0);
                    const uint2 b_hi4 = upper ? load_four_entries(sc_hi + table, group0 + gi, step_groups) : make_uint2(0, 0);
#pragma unroll
                    for (int c = 0; c < 4; ++c) {
                        const int within = gi + c < groups ? c : 0;
                        const int group = group0 + gi + within;
                        op[c].lower = lower + group * 32;
                        op[c].upper = upper_row + group * 32;
                        op[c].scale_lo = entry_of(s_lo4, within);
                        op[c].bias_lo = entry_of(b_lo4, within);
                        op[c].scale_hi = entry_of(s_hi4, within);
                        op[c].bias_hi = entry_of(b_hi4, within);
                        part[c][0] = part[c][1] = part[c][2] = part[c][3] = 0.0f;
                        into[c] = part[c];
                    }
                    if (upper) mma_groups<4, true>(op, bx0, bx1, x0, x1, into);
                    else mma_groups<4, false>(op, bx0, bx1, x0, x1, into);
#pragma unroll
                    for (int c = 0; c < 4; ++c)
                        if (gi + c < groups) {
#pragma unroll
                            for (int k = 0; k < 4; ++k) acc[k] += part[c][k];
                        }
#pragma unroll
                    for (int c = 0; c < 4; ++c) {
                        bx0[c] = nx0[c]; bx1[c] = nx1[c]; x0[c] = y0[c]; x1[c] = y1[c];
                    }
                }
            }
            // Hand back the items that end inside this tile.
            while (released < items2 && (released + 1) * lay.down_rows <= 16 * (tile + 1)) {
                const int it = first_down + released;
                if (it + slots < own_items) {
                    ptx::fence_proxy_async_smem();
                    __syncwarp();
                    if (lane == 0) ptx::mbar_arrive(&empty_bar[it % slots]);
                }
                ++released;
            }
            float* part = scratch + (size_t)(warp * 16) * 8;  // scratch[(warp * 16 + row) * 8 + column]
            *reinterpret_cast<float2*>(part + g * 8 + 2 * t) = make_float2(acc[0], acc[1]);
            *reinterpret_cast<float2*>(part + (g + 8) * 8 + 2 * t) = make_float2(acc[2], acc[3]);
            fused_compute_sync();
            const int rows_here = min(16, n2 - 16 * tile);
            for (int idx = threadIdx.x; idx < rows_here * M && met != kMeetLeft; idx += kFusedComputeThreads) {
                const int row = idx / M, m = idx - row * M;
                float v = 0.0f;
                for (int w = 0; w < kFusedComputeWarps; ++w) v += scratch[(w * 16 + row) * 8 + m];
                // The residual was fetched by thread (16 tile + row) * M + m, which is this one only in the
                // first tile; later tiles read it here.
                const size_t at = (size_t)m * H + row2 + 16 * tile + row;
                float extra = residual_value;
                if (tile > 0) extra = p.residual ? bf16_bits_to_f32(ptx::ld_global_dependent_u16(p.residual + at)) : 0.0f;
                p.out[at] = f32_to_bf16_bits(v + extra);
            }
            fused_compute_sync();
        }
        if (met == kMeetLast && next == 0 && (int)threadIdx.x < grid) fused_take_over(p.meeting, threadIdx.x, left_ctas, &left_count);
        ptx::fence_proxy_async_smem();  // the ring is filled again
        fused_compute_sync();
        if (threadIdx.x == 0) next_owner[next & 1] = next < left_count && !*abort_flag ? left_ctas[next] : -1;
        ptx::named_barrier_sync(2, kFusedThreads);  // the producer, too
        const int owner = next_owner[next & 1];
        if (owner < 0) break;
        first_down += items2;
        down_rows_of(owner);
        fetch_residual();
    }
    if (*abort_flag) ptx::drain_copies();
}

// Whether the eight-column kernel serves this problem.
inline bool fused_mlp_mma_applicable(const FusedMlpParams& p, int sm_count) {
    if (p.M < 1 || p.M > kFusedMmaMaxRows || sm_count < 1) return false;
    if (p.H < 512 || p.H % (64 * kFusedComputeWarps) || (p.H >> 6) / kFusedComputeWarps > kFusedMmaMaxGroups1) return false;
    if (p.I < 512 || p.I % (64 * kFusedComputeWarps)) return false;
    const FusedMlpLayout lay = fused_mlp_layout(p.H, p.I);
    if (lay.slots < 2 || lay.down_rows < 8 || lay.down_rows % 8) return false;
    if (((p.H + sm_count - 1) / sm_count + lay.down_rows - 1) / lay.down_rows > lay.slots) return false;
    if (16 * p.M > kFusedComputeThreads) return false;
    if (p.H % 256 || lay.item_bytes % 1024) return false;  // whole tensor-map boxes, swizzle-aligned items
    if (lay.total + 1024 > kFusedSmem || sm_count > kFusedMaxGrid) return false;
    const void* pointers[] = {p.x, p.gate_w, p.up_w, p.down_w, p.gate_s, p.gate_b, p.up_s, p.up_b, p.down_s, p.down_b,
                              p.hidden};
    for (const void* ptr : pointers)
        if (!aligned_to(ptr, 16)) return false;
    return true;
}

// Whether the fused kernel serves this problem on a device with `sm_count` SMs.
inline bool fused_mlp_applicable(const FusedMlpParams& p, int sm_count) {
    if (p.M < 1 || p.M > kFusedMaxRows || sm_count < 1 || sm_count > kFusedMaxGrid) return false;
    auto supported = [](int v) {  // two, four, eight or sixteen 512-column units
        return v >= 1024 && v <= 8192 && (v & (v - 1)) == 0;
    };
    if (!supported(p.H) || !supported(p.I) || p.H > 4096) return false;  // 8192 / 8192: two GEMV launches are as fast
    const FusedOneLayout lay = fused_one_layout(p.M, p.H, p.I, sm_count);
    if (lay.depth < 2 || lay.rows2_max * p.M > kFusedOneThreads) return false;
    const void* pointers[] = {p.x, p.gate_w, p.up_w, p.down_w, p.gate_s, p.gate_b, p.up_s, p.up_b, p.down_s, p.down_b,
                              p.hidden};
    for (const void* ptr : pointers)
        if (!aligned_to(ptr, 16)) return false;
    return true;
}

template <int kThreads>  // of a CTA, which also separates the kernels' static state
inline int launch_mlp_fused_kernel(void (*kernel)(const FusedMlpParams), int smem, const FusedMlpParams& params,
                                   int sm_count, int device, cudaStream_t stream) {
    static bool configured[64] = {};
    if (!configured[device]) {
        if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kFusedSmem) != cudaSuccess)
            return MT_ERR_LAUNCH;
        cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
        configured[device] = true;
    }
    cudaLaunchConfig_t config = {};
    config.gridDim = dim3(sm_count, 1, 1);
    config.blockDim = dim3(kThreads, 1, 1);
    config.dynamicSmemBytes = smem;
    config.stream = stream;
    cudaLaunchAttribute attrs[1];
    attrs[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attrs[0].val.programmaticStreamSerializationAllowed = 1;
    config.attrs = attrs;
    config.numAttrs = 1;
    return cudaLaunchKernelEx(&config, kernel, params) == cudaSuccess ? MT_OK : MT_ERR_LAUNCH;
}

// The slot of a launch into `stream`; -1 when there is none.
inline int meeting_slot_of(cudaStream_t stream) {
    static MeetingSlots* const slots = new MeetingSlots;  // never destroyed: launches may come late
    cudaStreamCaptureStatus status;
    unsigned long long capture = 0, id = 0;
    if (cudaStreamGetCaptureInfo(stream, &status, &capture) != cudaSuccess) return -1;
    if (status == cudaStreamCaptureStatusNone) return cudaStreamGetId(stream, &id) == cudaSuccess ? slots->of_stream(id) : -1;
    if (status != cudaStreamCaptureStatusActive) return -1;
    static thread_local char thread;  // a capturing stream does not tell its id (and asking ends the capture)
    return slots->of_capture(capture, reinterpret_cast<uintptr_t>(stream == cudaStreamPerThread ? (void*)&thread : (void*)stream));
}

// A slot on the current device.
inline bool meeting_place_of(int slot, FusedMeetingPlace& place) {
    static FusedMeetingSlot* first[64] = {};
    int device = 0;
    if (cudaGetDevice(&device) != cudaSuccess || device < 0 || device >= 64) return false;
    place.slot = __atomic_load_n(&first[device], __ATOMIC_ACQUIRE);
    if (!place.slot) {
        void* address = nullptr;
        if (cudaGetSymbolAddress(&address, g_fused_meetings) != cudaSuccess) return false;
        place.slot = static_cast<FusedMeetingSlot*>(address);
        __atomic_store_n(&first[device], place.slot, __ATOMIC_RELEASE);
    }
    place.slot += slot;
    return true;
}

// Every slot of the current device, which is idle, as it was in the beginning.
inline bool clear_meeting_places() {
    FusedMeetingPlace first;
    return meeting_place_of(0, first) && cudaMemset(first.slot, 0, sizeof(g_fused_meetings)) == cudaSuccess &&
           cudaDeviceSynchronize() == cudaSuccess;
}

// `launch` in its turn among the launches that share a slot although their streams do not: each begins behind the one before it.
template <typename Launch>
inline int launch_in_turn(int device, cudaStream_t stream, Launch&& launch) {
    static std::mutex mutex;
    static cudaEvent_t last[64] = {};
    const std::lock_guard<std::mutex> lock(mutex);
    if (!last[device] && cudaEventCreateWithFlags(&last[device], cudaEventDisableTiming) != cudaSuccess) {
        last[device] = nullptr;
        return MT_ERR_LAUNCH;
    }
    if (cudaStreamWaitEvent(stream, last[device], 0) != cudaSuccess) return MT_ERR_LAUNCH;  // an event not yet recorded holds nothing up
    const int rc = launch();
    if (rc == MT_OK && cudaEventRecord(last[device], stream) != cudaSuccess) cudaStreamSynchronize(stream);
    return rc;
}

// Caller has checked fused_mlp_applicable(), or fused_mlp_mma_applicable() when `mma` is set.
inline int launch_mlp_fused(FusedMlpParams params, int sm_count, bool mma, cudaStream_t stream) {
    int device = 0;
    cudaGetDevice(&device);
    if (device >= 64) return MT_ERR_DEVICE;
    const int slot = meeting_slot_of(stream);
    if (slot < 0 || !meeting_place_of(slot, params.meeting)) return MT_ERR_LAUNCH;
    auto start = [&](auto&& launch) { return slot == kMeetingShared ? launch_in_turn(device, stream, launch) : launch(); };
    if (mma) {
        if (!encode_weight_map(&params.gate_map, params.gate_w, params.H, params.I, kFusedItemRows) ||
            !encode_weight_map(&params.up_map, params.up_w, params.H, params.I, kFusedItemRows))
            return MT_ERR_LAUNCH;
        const int smem = fused_mlp_layout(params.H, params.I).total + 1024;
        return start([&] { return launch_mlp_fused_kernel<kFusedThreads>(affine_mlp_fused_mma_kernel, smem, params, sm_count, device, stream); });
    }
    const FusedOneLayout lay = fused_one_layout(params.M, params.H, params.I, sm_count);
    if (!encode_weight_map(&params.gate_map, params.gate_w, params.H, params.I, lay.tile1) ||
        !encode_weight_map(&params.up_map, params.up_w, params.H, params.I, lay.tile1) ||
        !encode_weight_map(&params.down_map, params.down_w, params.I, params.H, lay.tile2))
        return MT_ERR_LAUNCH;
    return start([&] { return launch_mlp_fused_kernel<kFusedOneThreads>(affine_mlp_fused_kernel, lay.total + 1024, params, sm_count, device, stream); });
}

}  // namespace mt
