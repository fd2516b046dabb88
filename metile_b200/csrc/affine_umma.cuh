// INT4 affine dequant-MMA on the 5th-generation tensor cores (tcgen05 + TMEM) for two rows and more (any
// row count in batch-invariant mode).
//
// Computes Y[M,N] = X[M,K] * dequant(W)[N,K]^T with the MLX layout the reference consumes
// (kernels/affine_qmv.py:25-51; shapes metile/backends/mlx_quantized.py:478-480), optionally
// fused gate|up with the SwiGLU epilogue g/(1+exp(-g))*u on un-rounded sums
// (kernels/affine_qmv.py:204-208) or the residual epilogue (:124-131).  It plays the role of the
// reference's multi-row matrix-unit path (metile/compiler/affine_quantized.py:7-99), which, like
// this kernel, rounds each dequantised weight to the 16-bit input type before the MMA
// (metile/codegen/msl_emitter.py:1413-1418) and accumulates in fp32.
//
// Shape of the computation ("swap-AB"): 128 weight rows are the MMA's M dimension (128 TMEM lanes), up to
// 128 activation rows (padded to a multiple of 16) its N dimension; K advances 16 elements per
// instruction.  With gate|up the 128 rows are 64 of gate and 64 of up, sixteen of each per TMEM quadrant, so
// that a tile is 64 outputs wide (the tile count decides how evenly the SMs are loaded: 5120 -> 27648 is 432
// tiles = 2.92 waves, where pairs of 128-row tiles were 1.46) and the two sums of an output meet by a shuffle.
//
//   weight warp    : TMA (per-CTA tiled load, 128B swizzle) of 128 rows x 128 B = four k-blocks (quantisation
//                    groups) per ring slot, and the scales and biases of the same slot by cp.async on the same
//                    barrier; read per thread from global memory those cost 32 L1 wavefronts per load
//   activation warp: [rows] x 128 columns (two k-blocks) per slot of a second ring by one 3-D TMA copy, straight
//                    into the swizzled B tiles; rows past M are zero-filled.  Four to eight slots deep: a copy
//                    takes longer than the multiplication of four k-blocks
//   dequant warps  : 16 warps, two groups that take the ring slots in turn, one thread per weight row and two
//                    k-blocks; nibbles -> bf16 (see dequant_word_bf16), stored to tensor memory as the A operand
//   MMA warps      : two, taking the slots in turn; one elected lane issues sixteen tcgen05.mma kind::f16 per slot
//                    (bf16 x bf16 -> fp32 in TMEM) and the tcgen05.commits that free what they read
//   epilogue warps : 4 warps read the accumulators while the next slice or tile is being multiplied: SwiGLU /
//                    residual, 16-byte bf16 stores along N
//
// CTAs are persistent (one per SM, tiles blockIdx, blockIdx + grid, ...).  Where the tiles cannot fill the SMs
// the K range of a tile is shared by a thread-block cluster instead (kCluster), whose CTAs store their sums into
// one another's shared memory.
//
// Determinism: an output is a sum over slices of the K range, in slice order.  In the fixed order (batch-invariant mode,
// a model's modules) a slice is one accumulator chain in ascending k (gate|up) or two, of its even and its odd pairs of
// k-blocks, added even + odd (plain); the slices are a function of (N, K, kernel family) only, and neither the tile's
// rows nor who computes a slice changes a bit, so a row's result does not depend on how many other rows are in the batch.
// A call that asks for no such thing has one chain per slice and the slices that suit its rows (umma_plan): at 2000 rows the
// MLP 2048 / 8192 takes 174 us instead of 231 (201 and 269 in a loop long enough to meet the power limit, where the SM
// clock settles at 1.50 and 1.66 GHz), at 128 rows 5120 / 27648 123 instead of 127.5 (such a loop).
//
// Measured in a replayed graph, against the kernel with two CTA-wide tiles, one hand-off per pair of k-blocks and a
// cluster sum read over DSMEM that this replaces (us): 16 rows gate|up 2048 -> 8192 10.9 -> 8.0, 8192 -> 2048 10.1 ->
// 7.6, 1536 -> 1536 5.0 -> 4.0, 1536 -> 32768 16.6 -> 9.8; 64 rows 13.1 -> 9.6, 11.6 -> 9.0, 6.3 -> 5.8, 21.1 -> 12.9;
// 128 rows 16.5 -> 12.7, 13.9 -> 12.0, 8.5 -> 7.5, 27.2 -> 21.4.  Long K: 445 -> 284 cycles per k-block at 16 rows
// (4.7 TB/s), 605 -> 442 at 128.  What is left: about 4.4 us per launch at any K (set-up 0.7, first weights 1, first
// dequantisation and MMA 1.3, epilogue and exit 1), and L2 traffic of the activations at many rows (each SM reads
// 64 KB of them per 16 KB of weights at 128 rows).
#pragma once

#include <cuda.h>

#include <algorithm>

#include "common.cuh"
#include "ptx.cuh"

namespace mt {

constexpr int kUmmaTileRows = 128;
constexpr int kUmmaBlockK = 64;         // one quantisation group
constexpr int kUmmaKBlocksPerSlot = 4;  // a ring slot holds 4 k-blocks: 128 B of packed nibbles per row
constexpr int kUmmaMaxRows = 128;       // activation rows of a tile

constexpr int kUmmaDequantWarps = 16;
constexpr int kUmmaWeightWarp = 16, kUmmaXWarp = 17, kUmmaMmaWarp = 18, kUmmaMmaWarp2 = 19;
constexpr int kUmmaEpilogueWarp = 20;   // 20..23: warp % 4 is the TMEM quadrant a warp can read
constexpr int kUmmaThreads = 24 * 32;

constexpr int kUmmaSlotBytes = kUmmaTileRows * 128;  // packed words of four k-blocks
constexpr int kUmmaTableBytes = kUmmaTileRows * 16;  // one 8-byte window of scales and one of biases per row
constexpr int kUmmaMaxSlots = 12;
constexpr int kUmmaMaxXSlots = 8;
constexpr int kUmmaStages = 2;                       // operand stages of four k-blocks, one per dequant group
constexpr int kUmmaBarrierBytes = 512;
constexpr int kUmmaOutBytes = 16 * 128 * 4;          // epilogue: sixteen activation rows of the tile, fp32
constexpr int kUmmaResidualPitch = 272;              // bytes of a residual row: 128 elements and the words at both ends
constexpr int kUmmaResidualSteps = 4;                // steps of sixteen rows whose residuals are in flight
constexpr int kUmmaResidualBytes = kUmmaResidualSteps * 16 * kUmmaResidualPitch;
constexpr int kUmmaSmemBytes = 227 * 1024;           // one CTA per SM, whatever the row count
// With few rows the kernel is as long as its start and its neighbours': a norm, a rotary embedding or a merge of attention splits
// finds room beside a CTA of 192 KB and 72 registers a thread (see the launch bounds), so that they overlap (decoding sixteen
// sequences of a four-block model, eight tokens: 1929 us with 227 KB and 80 registers, 1875 with 192 KB, 1843 with both).
__host__ __device__ constexpr int umma_smem_bytes(int npad) { return npad > 32 ? kUmmaSmemBytes : 192 * 1024; }
constexpr int kUmmaTmemCols = 512;                   // 256 accumulator columns, 2 x 128 operand columns
constexpr int kUmmaAColumn = 256;

// Activation slots of two k-blocks.
__host__ __device__ constexpr int umma_x_slots(int npad, bool windows, int side_bytes) {
    return npad > 64 ? (windows || side_bytes ? 4 : 5) : side_bytes ? 6 : 8;
}
// Ring depth: what the activation slots and the sums leave of shared memory.  With unaligned tables there are
// three more table entries than slots (see UmmaTables).
__host__ __device__ constexpr int umma_ring_slots(int npad, bool windows, int side_bytes) {
    const int x_bytes = umma_x_slots(npad, windows, side_bytes) * 2 * npad * 128;
    const int left = umma_smem_bytes(npad) - 1024 - kUmmaBarrierBytes - kUmmaOutBytes - side_bytes - x_bytes - (windows ? 3 * kUmmaTableBytes : 0);
    const int slots = left / (kUmmaSlotBytes + kUmmaTableBytes);
    return slots > kUmmaMaxSlots ? kUmmaMaxSlots : slots > 3 ? slots & ~1 : slots;  // even where there is a choice
}
// Warps that report a ring slot as done.  The two dequant groups take the slots in turn.  In a ring of even length a slot
// always belongs to the same group, which sees every phase of its barriers.  In an odd one it changes hands with
// every fill; a parity wait cannot tell a fill from the next but one, so there both groups wait for every fill, and the
// slot is filled again only when both have said that they saw it.
__host__ __device__ constexpr int umma_slot_reports(int ring_slots) { return ring_slots % 2 ? kUmmaDequantWarps : kUmmaDequantWarps / 2; }
static_assert(umma_ring_slots(128, false, 0) >= 3 && umma_ring_slots(128, true, 0) >= 3 && umma_ring_slots(64, true, 0) >= 4 &&
              umma_ring_slots(64, true, 64 * 512) >= 4 && umma_ring_slots(64, true, 8 * 16 * 512) >= 2 &&
              umma_ring_slots(64, true, 64 * 512 + kUmmaResidualBytes) >= 3 && umma_ring_slots(128, true, kUmmaResidualBytes) >= 3, "the ring is too short");
static_assert(8 * 32 * kUmmaTileRows * 4 <= umma_ring_slots(128, true, 0) * kUmmaSlotBytes + umma_x_slots(128, true, 0) * 2 * 128 * 128 &&
              8 * 24 * kUmmaTileRows * 4 <= umma_ring_slots(96, true, 0) * kUmmaSlotBytes + umma_x_slots(96, true, 0) * 2 * 96 * 128 &&
              8 * 20 * kUmmaTileRows * 4 <= umma_ring_slots(80, true, 0) * kUmmaSlotBytes + umma_x_slots(80, true, 0) * 2 * 80 * 128,
              "a cluster's slices (two per CTA at most) overlay both rings");
static_assert(8 * (2 * kUmmaMaxSlots + 2 * kUmmaStages + 2 * kUmmaMaxXSlots + 10) + 8 <= kUmmaBarrierBytes, "barrier area");

struct UmmaParams {
    CUtensorMap w_map[2];  // packed weights, uint32 [N, K/8], box {32, 128 rows (64 with gate|up)}, 128B swizzle
    CUtensorMap x_map;     // activations, bf16 [K/64][M][64], box {64, npad, 2}, 128B swizzle
    const void* x;
    const uint16_t* scales[2];
    const uint16_t* biases[2];
    const uint16_t* residual;
    uint16_t* out;
    int M, K, N;
    int slices;            // parts of the K range that are summed apart (see umma_slices)
    int chains;            // of a slice: one accumulator, or two for its even and its odd pairs of k-blocks
    int ksplit;            // CTAs of a cluster that share a tile's slices
    int row_tiles, act_tiles, npad;
    int unit_shift;        // log2 of the accumulator units in tensor memory
    int sum_bytes;         // shared memory of the running sum over a CTA's slices, or of the slices a cluster's CTA adds
    int side_bytes;        // that and the residuals in flight
    bool wide_out;         // rows of the output and the residual are 16-byte aligned
};

enum : unsigned int {
    kWaitRingEmpty = 0x101,
    kWaitRingFull = 0x102,
    kWaitAbEmpty = 0x103,
    kWaitAbFull = 0x104,
    kWaitAccFull = 0x105,
    kWaitAccEmpty = 0x107,
    kWaitXFull = 0x108,
    kWaitXEmpty = 0x109,
    kWaitTurn = 0x10A,
};

__device__ __forceinline__ uint32_t bf162_bits(__nv_bfloat162 v) { return *reinterpret_cast<uint32_t*>(&v); }
__device__ __forceinline__ __nv_bfloat162 bits_bf162(uint32_t v) { return *reinterpret_cast<__nv_bfloat162*>(&v); }

// Dequantisation reads a nibble as a SUBNORMAL bf16: the bits q (0..15) are the number q * 2^-133, and the
// bits 16q are q * 2^-129 (exponent field 0 or 1, one linear range), so masking alone makes numbers and one
// fma.rn.bf16x2 with the scale times 2^96 (2^92 for the upper nibble) and the bias times 2^-37 gives
// RN_bf16(scale * q + bias) * 2^-37: one rounding, and the power of two is taken out of the fp32 sums in the
// epilogue.  Ten instructions per word of eight weights; by way of 128 + q and a subtraction it took nineteen
// (445 -> 357 cycles per k-block at 16 rows).  Scales up to 2^31 and weights down to 2^-89 keep their bits.
constexpr uint32_t kDequantScalePair = 0x6D806F80u;  // bf16 2^92 (odd element: the bits hold 16q), 2^96 (even)
constexpr uint32_t kDequantBiasPair = 0x2D002D00u;   // bf16 2^-37 = 2^(96 - 133), twice
constexpr float kDequantUndo = 137438953472.0f;      // 2^37

// One packed word (8 nibbles) -> 8 bf16 weights in natural order: out[i] = (w_{2i}, w_{2i+1}) * 2^-37.
__device__ __forceinline__ void dequant_word_bf16(uint32_t w, __nv_bfloat162 scale2, __nv_bfloat162 bias2,
                                                  uint32_t* out) {
    const uint32_t even = w & 0x0F0F0F0Fu;  // bytes e0, e2, e4, e6
    const uint32_t odd = w & 0xF0F0F0F0u;   // bytes 16 e1, 16 e3, 16 e5, 16 e7
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        // Bytes (e_2i, 0, 16 e_2i+1, 0): a selector with its top bit set copies the sign of byte i, which is 0.
        const uint32_t select = (uint32_t)(i | ((8 | i) << 4) | ((4 + i) << 8) | ((8 | i) << 12));
        uint32_t pair;
        asm("prmt.b32 %0, %1, %2, %3;" : "=r"(pair) : "r"(even), "r"(odd), "r"(select));
        out[i] = bf162_bits(__hfma2(bits_bf162(pair), scale2, bias2));
    }
}

// What one CTA works on: its tiles, and its slices of their K range.
struct UmmaShare {
    int rank, first_tile, tile_step, tiles;
    int slices, slice_begin, slice_end, slots_total, slot_begin;
    int kblocks, kb_begin, nkb, nslots;
    // First slot of slice s, counted from this CTA's first slot.  Slices are whole ring slots (4 k-blocks) long.
    __device__ __forceinline__ int slice_slot(int s) const { return slots_total * s / slices - slot_begin; }
};

template <bool kCluster>
__device__ __forceinline__ UmmaShare umma_share(const UmmaParams& p) {
    UmmaShare w;
    w.rank = kCluster ? (int)blockIdx.x % p.ksplit : 0;  // equals the CTA's rank in its cluster
    w.first_tile = kCluster ? (int)blockIdx.x / p.ksplit : (int)blockIdx.x;
    w.tile_step = kCluster ? (int)gridDim.x / p.ksplit : (int)gridDim.x;
    w.tiles = p.row_tiles * p.act_tiles;
    w.kblocks = p.K / kUmmaBlockK;
    w.slices = p.slices;
    w.slots_total = (w.kblocks + kUmmaKBlocksPerSlot - 1) / kUmmaKBlocksPerSlot;
    w.slice_begin = kCluster ? p.slices * w.rank / p.ksplit : 0;
    w.slice_end = kCluster ? p.slices * (w.rank + 1) / p.ksplit : p.slices;
    w.slot_begin = kCluster ? w.slots_total * w.slice_begin / p.slices : 0;
    const int slot_end = kCluster ? w.slots_total * w.slice_end / p.slices : w.slots_total;
    w.nslots = slot_end - w.slot_begin;
    w.kb_begin = w.slot_begin * kUmmaKBlocksPerSlot;
    w.nkb = min(slot_end * kUmmaKBlocksPerSlot, w.kblocks) - w.kb_begin;
    return w;
}

// Whether slice s has a second pair of k-blocks at all (a chain of the odd pairs is otherwise never written).
__device__ __forceinline__ bool umma_slice_has_second(const UmmaShare& w, int s) {
    return w.nkb - w.slice_slot(s) * kUmmaKBlocksPerSlot > 2;
}

// Ring position of a running slot count.
struct RingCursor {
    int slot = 0;
    uint32_t phase = 0;
    __device__ __forceinline__ void advance(int slots) {
        if (++slot == slots) {
            slot = 0;
            phase ^= 1u;
        }
    }
};

// The weight row of TMEM lane r of a tile that starts at row n0 (rows past the end repeat the last).
template <bool kSwiglu>
__device__ __forceinline__ int umma_row(int n0, int r, int n_rows) {
    return min(n0 + (kSwiglu ? (r >> 5) * 16 + (r & 15) : r), n_rows - 1);
}

// The scales and biases of a tile's ring slots, copied by one warp: per slot one 8-byte asynchronous copy per row
// and table.  Where K % 256 == 0 and the arrays are 8-byte aligned that is exactly a slot's four entries.
// Otherwise a row's entries start `offset` (0..3) entries into an aligned 8-byte window, and a slot's entries lie in
// its own window and the one before, which the previous slot brought; the first slot of a tile brings window 0 in
// an entry of its own.  So the table ring has three entries more than the weight ring: entry E is overwritten
// ring + 3 entries later, when the slot after E's is known to be done, tile starts included while a tile has at
// least ring / 2 + 1 slots (umma_ring_in_use).  A window holds at least one entry of the row, so no copy
// touches memory outside the aligned 8 bytes around an array's ends, which the header asks to be readable.  (Copies that
// end with the array need a size each: 3 to 8 % of a launch over windows, and the same for the residuals' last word 5 to 18 %
// of many rows of an odd width.)  (Word by word -- up to 24 4-byte copies per lane and
// slot, each touching sixteen rows -- a slot took 1150 cycles at 106 rows, 6080 -> 11919.)
template <bool kWindows>
struct UmmaTables {
    const uint8_t* at[2][4];   // [scales, biases][rows 32 q + lane]: window of the tile's first slot
    uint32_t offsets;          // two bits for each of them

    template <bool kSwiglu>
    __device__ __forceinline__ void start_tile(const UmmaParams& p, const UmmaShare& w, int n0, int lane) {
        offsets = 0;
#pragma unroll
        for (int t = 0; t < 2; ++t)
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const uint16_t* base = (t ? p.biases : p.scales)[kSwiglu && lane >= 16];
                at[t][q] = reinterpret_cast<const uint8_t*>(base + (size_t)umma_row<kSwiglu>(n0, 32 * q + lane, p.N) * w.kblocks + w.kb_begin);
                if constexpr (kWindows) {
                    const uint32_t offset = (uint32_t)(reinterpret_cast<uintptr_t>(at[t][q]) >> 1) & 3u;
                    at[t][q] += offset ? 8 - 2 * offset : 0;
                    offsets |= offset << (8 * t + 2 * q);
                }
            }
    }
    // The first windows of a tile, for rows that do not start one.
    __device__ __forceinline__ void copy_head(uint8_t* entry, int lane) const {
        each([&](int t, int q, int offset) {
            if (offset) ptx::cp_async_8(entry + t * 1024 + (32 * q + lane) * 8, at[t][q] - 8);
        });
    }
    // The windows of slot `st`, of whose k-blocks `left` remain in the share.
    __device__ __forceinline__ void copy(int st, int left, uint8_t* entry, int lane) const {
        each([&](int t, int q, int offset) {
            if (!kWindows || offset == 0 || left >= 5 - offset) ptx::cp_async_8(entry + t * 1024 + (32 * q + lane) * 8, at[t][q] + 8 * st);
        });
    }

private:
    template <typename F>
    __device__ __forceinline__ void each(F&& f) const {
#pragma unroll
        for (int t = 0; t < 2; ++t)
#pragma unroll
            for (int q = 0; q < 4; ++q) f(t, q, (int)(offsets >> (8 * t + 2 * q)) & 3);
    }
};

// Slots of the weight ring that may be in flight: with unaligned tables, short tiles leave room for fewer.
__device__ __forceinline__ int umma_ring_in_use(bool windows, const UmmaShare& w, int ring_slots) {
    return windows ? min(ring_slots, w.nslots > 1 ? 2 * w.nslots - 2 : 1) : ring_slots;
}

// Sixteen accumulator columns of this warp's TMEM lanes, plus a second sixteen where there are some (eight at a
// time: the kernel has 80 registers a thread, and a kernel that spills even a few bytes has a stack, which
// cost about two microseconds per launch).
__device__ __forceinline__ void umma_read16(uint32_t acc, uint32_t acc2, bool second, float (&v)[16]) {
    uint32_t a[16];
    ptx::tmem_ld16(acc, a);
    ptx::tc_wait_ld16(a);
#pragma unroll
    for (int j = 0; j < 16; ++j) v[j] = __uint_as_float(a[j]);
    if (second) {
#pragma unroll
        for (int part = 0; part < 2; ++part) {
            uint32_t b[8];
            ptx::tmem_ld8(acc2 + 8 * part, b);
            ptx::tc_wait_ld8(b);
#pragma unroll
            for (int j = 0; j < 8; ++j) v[8 * part + j] += __uint_as_float(b[j]);
        }
    }
}

// ---- the sum over a cluster.  CTA `rank` finishes the activation rows rank, rank + ksplit, ... of the tile: every
// CTA stores its slices' sums for those rows into that CTA's shared memory, [slice][row / ksplit][TMEM lane] fp32,
// one cluster barrier, and the finishing CTA adds its own memory in slice order.  (With partial tiles left where they
// were computed and read over DSMEM, the remote loads and the second barrier they need took 6000 cycles of a
// 15000-cycle launch at 16 rows, 8192 -> 2048.)
__device__ __forceinline__ int umma_rows_per_cta(const UmmaParams& p) { return (p.npad + p.ksplit - 1) / p.ksplit; }

template <bool kSwiglu, bool kTwo>
__device__ __forceinline__ void umma_push_slices(const UmmaParams& p, const UmmaShare& w, uint32_t staging, uint32_t tmem, uint32_t unit_cols,
                                                 int rows, int thread) {
    const int rows_per_cta = umma_rows_per_cta(p);
    for (int s = w.slice_begin; s < w.slice_end; ++s) {
        const uint32_t acc = tmem + (uint32_t)(s - w.slice_begin) * unit_cols;
        const bool second = kTwo && umma_slice_has_second(w, s);
        uint32_t at = staging + 4u * (uint32_t)(s * rows_per_cta * kUmmaTileRows + thread);  // row / ksplit = 0
        int owner = 0;
        for (int c0 = 0; c0 < rows; c0 += 16) {
            float v[16];
            umma_read16(acc + c0, acc + c0 + (unit_cols >> 1), second, v);
#pragma unroll
            for (int j = 0; j < 16; ++j) {
                if (c0 + j < rows) ptx::st_cluster_f32(ptx::map_to_cta(at, (uint32_t)owner), v[j] * kDequantUndo);
                if (++owner == p.ksplit) {
                    owner = 0;
                    at += 4u * kUmmaTileRows;
                }
            }
        }
    }
}

template <bool kSwiglu>
__device__ __forceinline__ void umma_finish_rows(const UmmaParams& p, const UmmaShare& w, const float* staging, int m_base, int rows, int row_tile) {
    constexpr int kOut = kSwiglu ? 64 : 128;
    constexpr int kParts = kUmmaThreads / kOut;
    const int o = threadIdx.x % kOut, part = threadIdx.x / kOut;
    const int n = row_tile * kOut + o;
    if (n >= p.N) return;
    const int rows_per_cta = umma_rows_per_cta(p);
    const float* column = staging + (kSwiglu ? (o >> 4) * 32 + (o & 15) : o);  // TMEM lane of the output (of its gate)
    for (int i = part; w.rank + p.ksplit * i < rows; i += kParts) {
        const size_t at = (size_t)(m_base + w.rank + p.ksplit * i) * p.N + n;
        const uint32_t extra = !kSwiglu && p.residual ? ptx::ld_global_dependent_u16(p.residual + at) : 0u;
        const float* from = column + i * kUmmaTileRows;
        float first[8], second[8];
#pragma unroll
        for (int s = 0; s < 8; ++s) {
            first[s] = s < p.slices ? from[s * rows_per_cta * kUmmaTileRows] : 0.0f;
            second[s] = kSwiglu && s < p.slices ? from[s * rows_per_cta * kUmmaTileRows + 16] : 0.0f;
        }
#pragma unroll
        for (int s = 1; s < 8; ++s)
            if (s < p.slices) {
                first[0] += first[s];
                second[0] += second[s];
            }
        p.out[at] = f32_to_bf16_bits(kSwiglu ? swiglu_f32(first[0], second[0]) : first[0] + bf16_bits_to_f32(extra));
    }
}

// kWindows: the four scales (biases) of a slot are not one aligned 8-byte vector (see UmmaTables).  A kernel of its own,
// because every instruction that the dequantising warps do not issue counts: with the layout as a run-time condition 512
// rows 1536 -> 8960, gate|up, took 37.6 us, now 34.0; 2000 rows 2048 -> 8192 153, now 144; 16 rows 8192 -> 2048 8.5, now 8.2.
// kFew: 72 registers a thread instead of 80, for up to 32 rows (umma_smem_bytes).  With windows a launch loses 2 to 3 % by it.
// kTwo: two chains per slice.  As a run-time condition it cost launches at 512 rows 2 % (the 24 of a prompt through four blocks, with
// the bounds of kFew: 3.5 us of 548).
template <bool kSwiglu, bool kCluster, bool kWindows, bool kFew, bool kTwo>
__global__ void __launch_bounds__(kFew ? kUmmaThreads + 128 : kUmmaThreads, 1) affine_umma_kernel(const __grid_constant__ UmmaParams p) {
    constexpr int kOut = kSwiglu ? 64 : 128;  // outputs per tile
    extern __shared__ uint8_t smem_raw[];
    // Aligned by offsetting the array itself (not by rounding a generic address), so that the compiler
    // still knows these are shared-memory addresses and emits shared loads and stores.
    uint8_t* smem = smem_raw + ((1024u - (ptx::smem_u32(smem_raw) & 1023u)) & 1023u);
    const int npad = p.npad;
    const UmmaShare w = umma_share<kCluster>(p);
    const int ring_space = umma_ring_slots(npad, kWindows, p.side_bytes);
    const int ring_slots = umma_ring_in_use(kWindows, w, ring_space);
    const int table_slots = kWindows ? ring_slots + 3 : ring_slots;
    const int x_slots = umma_x_slots(npad, kWindows, p.side_bytes), x_slot_bytes = 2 * npad * 128;
    uint8_t* ring = smem;
    uint8_t* x_tiles = ring + ring_space * kUmmaSlotBytes;
    uint8_t* tables = x_tiles + x_slots * x_slot_bytes;
    float* out_tile = reinterpret_cast<float*>(tables + (kWindows ? ring_space + 3 : ring_space) * kUmmaTableBytes);
    float* sum_tile = out_tile + kUmmaOutBytes / 4;
    uint8_t* residual_ring = reinterpret_cast<uint8_t*>(sum_tile) + p.sum_bytes;
    uint64_t* ring_full = reinterpret_cast<uint64_t*>(reinterpret_cast<uint8_t*>(sum_tile) + p.side_bytes);
    uint64_t* ring_empty = ring_full + kUmmaMaxSlots;
    uint64_t* a_full = ring_empty + kUmmaMaxSlots;
    uint64_t* stage_empty = a_full + kUmmaStages;
    uint64_t* x_full = stage_empty + kUmmaStages;
    uint64_t* x_empty = x_full + kUmmaMaxXSlots;
    uint64_t* turn = x_empty + kUmmaMaxXSlots;
    uint64_t* acc_full = turn + 2;
    uint64_t* acc_empty = acc_full + 4;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_empty + 4);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

    const int warp = __shfl_sync(0xFFFFFFFFu, threadIdx.x >> 5, 0);  // the same for the whole warp, and known to be
    const int lane = threadIdx.x & 31;
    // Accumulator units: one slice's sums, in one chain or in two halves of the unit.
    const uint32_t unit_mask = (1u << p.unit_shift) - 1u, unit_cols = (uint32_t)kUmmaAColumn >> p.unit_shift;
    const uint32_t second_col = unit_cols >> 1;

    if (threadIdx.x == 0) {
        for (int i = 0; i < ring_slots; ++i) {
            ptx::mbar_init(&ring_full[i], 1 + 32);  // the weight copy, and every lane's table copies
            ptx::mbar_init(&ring_empty[i], umma_slot_reports(ring_slots));
        }
        for (int i = 0; i < kUmmaStages; ++i) {
            ptx::mbar_init(&a_full[i], kUmmaDequantWarps / 2);
            ptx::mbar_init(&stage_empty[i], 1);
        }
        for (int i = 0; i < x_slots; ++i) {
            ptx::mbar_init(&x_full[i], 1);
            ptx::mbar_init(&x_empty[i], 1);
        }
        for (int i = 0; i < 2; ++i) ptx::mbar_init(&turn[i], 1);
        for (int i = 0; i < 4; ++i) {
            ptx::mbar_init(&acc_full[i], 2);
            ptx::mbar_init(&acc_empty[i], 4);
        }
        *abort_flag = 0;
        ptx::mbar_fence_init();
    }
    if (warp == kUmmaMmaWarp) {
        ptx::tmem_alloc(tmem_slot, kUmmaTmemCols);
        ptx::tmem_relinquish();
    }
    ptx::tc_fence_before_sync();
    __syncthreads();
    ptx::tc_fence_after_sync();
    const uint32_t tmem_base = *tmem_slot;
    if constexpr (kCluster) ptx::cluster_arrive();  // this CTA's shared memory can be written (see the end)
    // Programmatic dependent launch: the next kernel of the stream may begin its own set-up and
    // weight prefetch while this one is still running.  Only the weights (which no kernel writes)
    // are touched before griddep_wait(); activations, residual and outputs come after it.
    ptx::griddep_launch_dependents();

    if (warp == kUmmaWeightWarp) {
        // ------------------------------------------------------------------ packed weights by TMA, their tables
        // The whole warp runs the loop (see the MMA issuers); one elected lane issues the TMA copies, and every
        // lane copies the scales and biases of four rows.
        if (ptx::elect_one()) {
            ptx::prefetch_tensor_map(&p.w_map[0]);
            if (kSwiglu) ptx::prefetch_tensor_map(&p.w_map[1]);
        }
        __syncwarp();
        UmmaTables<kWindows> copies;
        RingCursor at, table_at;
        bool alive = true;
        for (int tile = w.first_tile; tile < w.tiles && alive; tile += w.tile_step) {
            const int n0 = tile / p.act_tiles * kOut;
            copies.template start_tile<kSwiglu>(p, w, n0, lane);
            for (int st = 0; st < w.nslots; ++st, at.advance(ring_slots)) {
                if (!ptx::mbar_wait(&ring_empty[at.slot], at.phase ^ 1u, abort_flag, kWaitRingEmpty)) { alive = false; break; }
                __syncwarp();
                if (ptx::elect_one()) {
                    ptx::mbar_expect_tx(&ring_full[at.slot], kUmmaSlotBytes);
                    uint8_t* slot = ring + at.slot * kUmmaSlotBytes;
                    const int word = w.kb_begin * 8 + st * 32;
                    ptx::tma_load_2d(slot, &p.w_map[0], word, n0, &ring_full[at.slot]);
                    if (kSwiglu) ptx::tma_load_2d(slot + kUmmaSlotBytes / 2, &p.w_map[1], word, n0, &ring_full[at.slot]);
                }
                __syncwarp();
                if (kWindows && st == 0) {
                    copies.copy_head(tables + table_at.slot * kUmmaTableBytes, lane);
                    table_at.advance(table_slots);
                }
                copies.copy(st, w.nkb - st * kUmmaKBlocksPerSlot, tables + table_at.slot * kUmmaTableBytes, lane);
                table_at.advance(table_slots);
                ptx::cp_async_arrive(&ring_full[at.slot]);
            }
        }
        ptx::cp_async_wait_all();
        if (*abort_flag) ptx::drain_copies();
    } else if (warp == kUmmaXWarp) {
        // ------------------------------------------------------------------ activation tiles by TMA
        if (ptx::elect_one()) ptx::prefetch_tensor_map(&p.x_map);
        __syncwarp();
        ptx::griddep_wait();  // the activations are the preceding kernel's output
        RingCursor at;
        bool alive = true;
        for (int tile = w.first_tile; tile < w.tiles && alive; tile += w.tile_step) {
            const int m0 = tile % p.act_tiles * npad;
            for (int kb = 0; kb < w.nkb; kb += 2, at.advance(x_slots)) {
                if (!ptx::mbar_wait(&x_empty[at.slot], at.phase ^ 1u, abort_flag, kWaitXEmpty)) { alive = false; break; }
                __syncwarp();
                if (ptx::elect_one()) {
                    // A k-block past the end of the matrix is filled with zeros and never multiplied.
                    ptx::mbar_expect_tx(&x_full[at.slot], (uint32_t)x_slot_bytes);
                    ptx::tma_load_3d(x_tiles + at.slot * x_slot_bytes, &p.x_map, 0, m0, w.kb_begin + kb, &x_full[at.slot]);
                }
                __syncwarp();
            }
        }
        if (*abort_flag) ptx::drain_copies();
    } else if (warp == kUmmaMmaWarp || warp == kUmmaMmaWarp2) {
        // ------------------------------------------------------------------ MMA issuers
        // Two warps take the slots in turn; each has done its waiting (130 cycles a wait even when it is already
        // satisfied) by the time the other one passes it the turn, so that the pipe does not run dry between
        // slots.  All of a warp's lanes run the loop and one elected lane issues: with the loop under
        // `lane == 0` the operands are not in uniform registers and an MMA took 66 cycles to issue.
        const int mine = warp == kUmmaMmaWarp ? 0 : 1;
        const uint32_t idesc = ptx::umma_idesc_bf16(kUmmaTileRows, npad);
        const uint64_t desc0 = ptx::smem_desc_k_major_sw128(ptx::smem_u32(x_tiles));
        const uint32_t a_tmem = tmem_base + kUmmaAColumn + mine * 128;
        uint32_t count = 0;
        RingCursor x_at;
        uint32_t q = 0;  // slices so far
        bool alive = true;
        for (int tile = w.first_tile; tile < w.tiles && alive; tile += w.tile_step) {
            for (int s = w.slice_begin; s < w.slice_end && alive; ++s, ++q) {
                const uint32_t unit = q & unit_mask;
                const uint32_t d_tmem = tmem_base + unit * unit_cols;
                const int begin = w.slice_slot(s), end = w.slice_slot(s + 1);
                for (int st = begin; st < end && alive; ++st, ++count) {
                    const int valid = w.nkb - st * kUmmaKBlocksPerSlot;  // fewer than four only at a ragged end
                    const RingCursor first = x_at;
                    x_at.advance(x_slots);
                    const RingCursor second = x_at;
                    if (valid > 2) x_at.advance(x_slots);
                    if ((int)(count & 1u) != mine) continue;
                    // A parity wait is only right when the phase before the awaited one is known to be over.  For the
                    // accumulators that is the previous slice's own wait: with two units and more it lies at least two slots
                    // back, and this warp has had the turn since; with one unit and a slice of one slot it is the other
                    // warp's for the slot just before, so there the turn comes first.
                    const uint32_t acc_parity = ((q >> p.unit_shift) & 1u) ^ 1u;
                    const bool acc_first = st == begin && unit_mask != 0, acc_last = st == begin && unit_mask == 0;
                    alive = (!acc_first || ptx::mbar_wait_spin(&acc_empty[unit], acc_parity, abort_flag, kWaitAccEmpty)) &&
                            ptx::mbar_wait_spin(&x_full[first.slot], first.phase, abort_flag, kWaitXFull) &&
                            (valid <= 2 || ptx::mbar_wait_spin(&x_full[second.slot], second.phase, abort_flag, kWaitXFull)) &&
                            ptx::mbar_wait_spin(&a_full[mine], (count >> 1) & 1u, abort_flag, kWaitAbFull) &&
                            (count == 0 || ptx::mbar_wait_spin(&turn[mine], ((count - 1) >> 1) & 1u, abort_flag, kWaitTurn)) &&
                            (!acc_last || ptx::mbar_wait_spin(&acc_empty[unit], acc_parity, abort_flag, kWaitAccEmpty));
                    if (!alive) break;
                    __syncwarp();
                    ptx::tc_fence_after_sync();
                    if (ptx::elect_one()) {
#pragma unroll
                        for (int kb = 0; kb < kUmmaKBlocksPerSlot; ++kb) {
                            if (kb >= valid) break;
                            const int x_slot = kb < 2 ? first.slot : second.slot;
                            const uint64_t b_desc = desc0 + (uint64_t)((x_slot * x_slot_bytes + (kb & 1) * npad * 128) >> 4);
                            const uint32_t d = kTwo && kb >= 2 ? d_tmem + second_col : d_tmem;
                            const bool starts = st == begin && (kb == 0 || (kb == 2 && kTwo));
#pragma unroll
                            for (int ks = 0; ks < kUmmaBlockK / 16; ++ks)  // the first MMA into an accumulator overwrites it
                                ptx::umma_ts(d, a_tmem + kb * 32 + ks * 8, b_desc + (uint64_t)(ks * 2), idesc, starts && ks == 0 ? 0u : 1u);
                            if (kb == 1 || (kb == 0 && valid == 1)) ptx::umma_commit(&x_empty[first.slot]);
                        }
                        ptx::tc_fence_before_sync();
                        ptx::mbar_arrive(&turn[mine ^ 1]);
                        if (valid > 2) ptx::umma_commit(&x_empty[second.slot]);
                        ptx::umma_commit(&stage_empty[mine]);
                        // Both issuers report the slice: the one of its last slot, and the one of the slot before it.
                        if (st + 2 >= end) ptx::umma_commit(&acc_full[unit]);
                        if (end - begin == 1) ptx::umma_commit(&acc_full[unit]);
                    }
                    __syncwarp();
                }
            }
        }
    } else if (warp >= kUmmaEpilogueWarp) {
        // ------------------------------------------------------------------ epilogue
        const int quadrant = warp & 3;
        const uint32_t lane_base = (uint32_t)(quadrant * 32) << 16;
        constexpr int kPitch = kSwiglu ? 80 : 128;  // floats per staged row; 80: both half-warps' rows without conflicts
        constexpr int kVectors = kOut / 8;          // 16-byte vectors of an output row
        const int thread = quadrant * 32 + lane;    // of the four warps
        const int my_slices = w.slice_end - w.slice_begin;
        ptx::griddep_wait();  // the residual is, and the output may still be read by, a preceding kernel
        uint32_t q = 0;       // slices so far
        bool alive = true;
        // Waits for accumulator unit `index`; false in the whole warp when it gave up.
        auto wait_unit = [&](uint32_t index) {
            alive = __all_sync(0xFFFFFFFFu, alive && ptx::mbar_wait(&acc_full[index & unit_mask], (index >> p.unit_shift) & 1u,
                                                                    abort_flag, kWaitAccFull));
            ptx::tc_fence_after_sync();
            return alive;
        };
        auto release_unit = [&](uint32_t index) {
            ptx::tc_fence_before_sync();
            __syncwarp();
            if (lane == 0) ptx::mbar_arrive(&acc_empty[index & unit_mask]);
        };
        auto unit_address = [&](uint32_t index) { return tmem_base + lane_base + (index & unit_mask) * unit_cols; };
        for (int tile = w.first_tile; tile < w.tiles && alive; tile += w.tile_step) {
            if constexpr (kCluster) {
                for (int s = 0; s < my_slices; ++s) wait_unit(q + s);
                break;  // a cluster has one tile; its sums are exchanged at the end
            } else {
                const int row_tile = tile / p.act_tiles;
                const int m0 = (tile - row_tile * p.act_tiles) * npad;
                const int rows = min(npad, p.M - m0);
                const int n_tile = row_tile * kOut;
                // The residuals of four steps of sixteen activation rows are on their way by asynchronous copies, the first
                // ones while the tile is still being multiplied; held in registers one step ahead they cost a memory
                // round trip per step (445 rows 1024 -> 50240: 115 us against 86, and 67 without a residual).  Where
                // rows are 16-byte aligned, 16 bytes per copy; else the words that hold the row's elements: warp q has
                // rows 4 q .. 4 q + 3 of a step, a lane words `lane` and `lane + 32`, one lane per row a 65th.
                const bool has_residual = !kSwiglu && p.residual != nullptr;
                auto odd_start = [&](const uint16_t* base, int m) {  // whether the tile's row m starts in the middle of a word
                    return (int)((reinterpret_cast<uintptr_t>(base) >> 1) + (uint32_t)(m0 + m) * (uint32_t)p.N) & 1;
                };
                auto request_residual = [&](int c0) {
                    if constexpr (!kSwiglu) {
                        if (!has_residual) return;
                        uint8_t* step = residual_ring + (c0 / 16 % kUmmaResidualSteps) * (16 * kUmmaResidualPitch);
                        if (c0 < rows && p.wide_out) {
#pragma unroll
                            for (int i = 0; i < 2; ++i) {
                                const int at = thread + 128 * i, j = at / kVectors, n = n_tile + at % kVectors * 8;
                                if (c0 + j < rows && n < p.N)
                                    ptx::cp_async_16(step + j * kUmmaResidualPitch + at % kVectors * 16, p.residual + (size_t)(m0 + c0 + j) * p.N + n);
                            }
                        } else if (c0 < rows) {
                            auto copy_word = [&](int j, int word) {
                                const int n = n_tile + 2 * word - odd_start(p.residual, c0 + j);  // n, n + 1: at least one is in the row
                                if (c0 + j < rows && n < p.N)
                                    ptx::cp_async_4(step + j * kUmmaResidualPitch + 4 * word, p.residual + (size_t)(m0 + c0 + j) * p.N + n);
                            };
#pragma unroll
                            for (int i = 0; i < 8; ++i) copy_word(quadrant * 4 + (i >> 1), lane + 32 * (i & 1));
                            if (lane < 4 && odd_start(p.residual, c0 + quadrant * 4 + lane)) copy_word(quadrant * 4 + lane, 64);
                        }
                        ptx::cp_async_commit();
                    }
                };
#pragma unroll
                for (int i = 0; i < kUmmaResidualSteps; ++i) request_residual(16 * i);

                // Slices that the final pass does not read itself go to the running sum, which holds all padded rows.
                const int direct = kSwiglu && my_slices == 2 ? 2 : 1;
                float* sums = sum_tile + thread;
                for (int s = 0; s < my_slices - direct; ++s, ++q) {
                    if (!wait_unit(q)) break;
                    const uint32_t acc = unit_address(q);
                    const bool second = kTwo && umma_slice_has_second(w, s);
                    for (int c0 = 0; c0 < rows; c0 += 16) {
                        float v[16];
                        umma_read16(acc + c0, acc + c0 + second_col, second, v);
#pragma unroll
                        for (int half = 0; half < 2; ++half) {
                            float before[8];
#pragma unroll
                            for (int j = 0; j < 8; ++j) before[j] = s > 0 ? sums[(c0 + 8 * half + j) * kUmmaTileRows] : 0.0f;
#pragma unroll
                            for (int j = 0; j < 8; ++j)
                                sums[(c0 + 8 * half + j) * kUmmaTileRows] = s > 0 ? before[j] + v[8 * half + j] : v[8 * half + j];
                        }
                    }
                    release_unit(q);
                }
                if (!alive) break;

                // The final pass: the last slice (or its two chains) after the running sum of the earlier ones, or both of
                // gate|up's two slices.
                if (!wait_unit(q) || (direct == 2 && !wait_unit(q + 1))) break;
                const uint32_t acc = unit_address(q);
                const bool second = kSwiglu ? direct == 2 : kTwo && umma_slice_has_second(w, w.slice_end - 1);
                const uint32_t acc2 = kSwiglu ? unit_address(q + 1) : acc + second_col;
                const bool earlier = my_slices > direct;
                // Sixteen activation rows at a time through shared memory, so that an output row leaves as 16-byte
                // vectors.  Stored straight from the registers (two bytes per lane and row, residual read the same
                // way) a 128 x 128 tile took 13000 to 40000 cycles, more than the multiplication of its operands.
                // Plain: lane = output.  Gate|up: lanes 0..15 hold gate, 16..31 up of the same sixteen outputs;
                // after one exchange per column pair the lower half finishes the even column, the upper the odd one.
                const bool upper = lane >= 16;
                for (int c0 = 0; c0 < rows; c0 += 16) {
                    float v[16];
                    umma_read16(acc + c0, acc2 + c0, second, v);
                    if (earlier) {
#pragma unroll
                        for (int j = 0; j < 16; ++j) v[j] = sums[(c0 + j) * kUmmaTileRows] + v[j];
                    }
                    if constexpr (kSwiglu) {
                        float gate[8], up[8], value[8];
#pragma unroll
                        for (int j = 0; j < 8; ++j) {
                            const float mine = (upper ? v[2 * j + 1] : v[2 * j]) * kDequantUndo;
                            const float other = __shfl_xor_sync(0xFFFFFFFFu, (upper ? v[2 * j] : v[2 * j + 1]) * kDequantUndo, 16);
                            gate[j] = upper ? other : mine;
                            up[j] = upper ? mine : other;
                        }
                        swiglu8_f32(gate, up, value);
                        if (c0 > 0) ptx::named_barrier_sync(1, 128);  // the rows staged before have been read
#pragma unroll
                        for (int j = 0; j < 8; ++j) out_tile[(2 * j + (upper ? 1 : 0)) * kPitch + quadrant * 16 + (lane & 15)] = value[j];
                    } else {
                        if (c0 > 0) ptx::named_barrier_sync(1, 128);
#pragma unroll
                        for (int j = 0; j < 16; ++j) out_tile[j * kPitch + thread] = v[j] * kDequantUndo;
                        ptx::cp_async_wait_group<kUmmaResidualSteps - 1>();  // this step's residuals
                    }
                    const uint8_t* residual_step = residual_ring + (c0 / 16 % kUmmaResidualSteps) * (16 * kUmmaResidualPitch);
                    ptx::named_barrier_sync(1, 128);
                    if (p.wide_out) {
#pragma unroll
                        for (int i = 0; i < kOut / 64; ++i) {
                            const int at = thread + 128 * i, j = at / kVectors, n = n_tile + at % kVectors * 8;
                            if (c0 + j < rows && n < p.N) {
                                const float4 lo = *reinterpret_cast<const float4*>(out_tile + j * kPitch + at % kVectors * 8);
                                const float4 hi = *reinterpret_cast<const float4*>(out_tile + j * kPitch + at % kVectors * 8 + 4);
                                uint4 packed;
                                if (has_residual) {
                                    const uint4 r = *reinterpret_cast<const uint4*>(residual_step + j * kUmmaResidualPitch + at % kVectors * 16);
                                    packed.x = pack_bf16x2(lo.x + bf16_lo(r.x), lo.y + bf16_hi(r.x));
                                    packed.y = pack_bf16x2(lo.z + bf16_lo(r.y), lo.w + bf16_hi(r.y));
                                    packed.z = pack_bf16x2(hi.x + bf16_lo(r.z), hi.y + bf16_hi(r.z));
                                    packed.w = pack_bf16x2(hi.z + bf16_lo(r.w), hi.w + bf16_hi(r.w));
                                } else {
                                    packed = make_uint4(pack_bf16x2(lo.x, lo.y), pack_bf16x2(lo.z, lo.w), pack_bf16x2(hi.x, hi.y),
                                                        pack_bf16x2(hi.z, hi.w));
                                }
                                *reinterpret_cast<uint4*>(p.out + (size_t)(m0 + c0 + j) * p.N + n) = packed;
                            }
                        }
                        request_residual(c0 + 16 * kUmmaResidualSteps);
                    } else if constexpr (!kSwiglu) {
                        // All reads before the first store, with no branch among them: a step is bounded by shared
                        // memory's latency (445 rows 1024 -> 50243: 84 us, 132 as one branching loop over the words).
                        uint32_t packed[8];
                        auto element_pair = [&](int j, int e, int residual_odd) {  // elements e, e + 1 of a row; one may lie outside the tile
                            float a = out_tile[j * kPitch + e], b = out_tile[j * kPitch + e + 1];
                            if (has_residual) {
                                const uint16_t* r = reinterpret_cast<const uint16_t*>(residual_step + j * kUmmaResidualPitch) + e + residual_odd;
                                a += bf16_bits_to_f32(r[0]);
                                b += bf16_bits_to_f32(r[1]);
                            }
                            return pack_bf16x2(a, b);
                        };
#pragma unroll
                        for (int i = 0; i < 8; ++i) {
                            const int j = quadrant * 4 + (i >> 1);
                            packed[i] = element_pair(j, 2 * (lane + 32 * (i & 1)) - odd_start(p.out, c0 + j), odd_start(p.residual, c0 + j));
                        }
#pragma unroll
                        for (int i = 0; i < 8; ++i) {
                            const int m = c0 + quadrant * 4 + (i >> 1), e = 2 * (lane + 32 * (i & 1)) - odd_start(p.out, m), n = n_tile + e;
                            uint16_t* to = p.out + (size_t)(m0 + m) * p.N + n;
                            const bool low = m < rows && e >= 0 && n < p.N, high = m < rows && n + 1 < p.N;
                            if (low && high) *reinterpret_cast<uint32_t*>(to) = packed[i];
                            if (low && !high) to[0] = (uint16_t)packed[i];
                            if (high && !low) to[1] = (uint16_t)(packed[i] >> 16);
                        }
                        // The last element of a row that starts in the middle of a word.
                        const int last_row = quadrant * 4 + (lane & 3);
                        if (lane < 4 && c0 + last_row < rows && n_tile + 127 < p.N && odd_start(p.out, c0 + last_row))
                            p.out[(size_t)(m0 + c0 + last_row) * p.N + n_tile + 127] = (uint16_t)element_pair(last_row, 127, odd_start(p.residual, c0 + last_row));
                        __syncwarp();  // the copies below overwrite what other lanes read
                        request_residual(c0 + 16 * kUmmaResidualSteps);
                    } else {
                        const int o = thread % kOut, n = n_tile + o;
                        for (int j = thread / kOut; j < 16 && c0 + j < rows; j += 128 / kOut)
                            if (n < p.N) p.out[(size_t)(m0 + c0 + j) * p.N + n] = f32_to_bf16_bits(out_tile[j * kPitch + o]);
                    }
                }
                for (int s = 0; s < direct; ++s, ++q) release_unit(q);
                ptx::named_barrier_sync(1, 128);  // before the next tile stages its rows
            }
        }
    } else {
        // ------------------------------------------------------------------ dequant warps
        // Two groups of eight warps take the slots in turn, each into its own operand stage, so that one group
        // dequantises (the logic pipe is busy: 48 half-rate instructions per k-block and thread) while the
        // other one waits, stores and reports.  A thread handles one row of two of the slot's k-blocks.
        const int quadrant = warp & 3, half = (warp >> 2) & 1, group = warp >> 3;
        const int r = quadrant * 32 + lane;            // TMEM lane
        // Its row of the slot: the 64 gate rows come first, then the 64 up rows.
        const int row = kSwiglu ? (lane >> 4) * 64 + quadrant * 16 + (lane & 15) : r;
        const uint32_t a_lane = tmem_base + ((uint32_t)(quadrant * 32) << 16) + kUmmaAColumn + group * 128 + half * 64;
        const uint16_t* table_base[2] = {p.scales[kSwiglu && lane >= 16], p.biases[kSwiglu && lane >= 16]};
        const bool even_ring = (ring_slots & 1) == 0;
        RingCursor at, table_at;
        uint32_t count = 0, use = 0;  // slots seen, slots handled
        bool alive = true;
        for (int tile = w.first_tile; tile < w.tiles && alive; tile += w.tile_step) {
            // Position of this thread's first entry in the eight entries of the window before and the slot's own.
            // (kb_begin and a slot are multiples of four entries, so it is the same for all slots of a row.)
            uint32_t position[2] = {4u + 2u * half, 4u + 2u * half};
            if (kWindows) {
                const size_t entry = (size_t)umma_row<kSwiglu>(tile / p.act_tiles * kOut, r, p.N) * w.kblocks;
#pragma unroll
                for (int t = 0; t < 2; ++t) {
                    const uint32_t offset = (uint32_t)(reinterpret_cast<uintptr_t>(table_base[t] + entry) >> 1) & 3u;
                    position[t] = (offset ? offset : 4u) + 2u * half;
                }
                table_at.advance(table_slots);  // the first windows
            }
            for (int st = 0; st < w.nslots; ++st, ++count, at.advance(ring_slots), table_at.advance(table_slots)) {
                if ((count & 1u) != (uint32_t)group && even_ring) continue;
                if (!ptx::mbar_wait(&ring_full[at.slot], at.phase, abort_flag, kWaitRingFull)) { alive = false; break; }
                if ((count & 1u) != (uint32_t)group) {
                    __syncwarp();
                    if (lane == 0) ptx::mbar_arrive(&ring_empty[at.slot]);
                    continue;
                }
                const uint8_t* slot = ring + at.slot * kUmmaSlotBytes + row * 128;
                uint32_t pair[2];  // the scales and the biases of this thread's two k-blocks
                const uint8_t* own = tables + table_at.slot * kUmmaTableBytes + r * 8;
                if (kWindows) {
                    const uint8_t* before = table_at.slot > 0 ? own - kUmmaTableBytes : own + (table_slots - 1) * kUmmaTableBytes;
#pragma unroll
                    for (int t = 0; t < 2; ++t) {
                        const uint32_t word = position[t] >> 1;  // 0, 1: the window before; 2, 3: the slot's own
                        const uint8_t* low = (word < 2 ? before + 4 * word : own + 4 * (word - 2)) + t * 1024;
                        const uint8_t* high = word < 1 ? low + 4 : own + 4 * (word - 1) + t * 1024;  // read in odd positions only
                        const uint32_t first = *reinterpret_cast<const uint32_t*>(low);
                        pair[t] = position[t] & 1u ? __funnelshift_r(first, *reinterpret_cast<const uint32_t*>(high), 16) : first;
                    }
                } else {
                    pair[0] = *reinterpret_cast<const uint32_t*>(own + 4 * half);
                    pair[1] = *reinterpret_cast<const uint32_t*>(own + 4 * half + 1024);
                }
#pragma unroll
                for (int kb = 0; kb < 2; ++kb) {
                    const int j = 2 * half + kb;       // 32 B of the row: chunks 2j and 2j + 1, XOR-swizzled by the row
                    const uint4 w_lo = *reinterpret_cast<const uint4*>(slot + (((2 * j) ^ (row & 7)) << 4));
                    const uint4 w_hi = *reinterpret_cast<const uint4*>(slot + (((2 * j + 1) ^ (row & 7)) << 4));
                    const uint32_t both = kb == 0 ? 0x1010u : 0x3232u;
                    const __nv_bfloat162 scale2 = __hmul2(bits_bf162(__byte_perm(pair[0], 0u, both)), bits_bf162(kDequantScalePair));
                    const __nv_bfloat162 bias2 = __hmul2(bits_bf162(__byte_perm(pair[1], 0u, both)), bits_bf162(kDequantBiasPair));
                    uint32_t wq[32];
                    const uint32_t words8[8] = {w_lo.x, w_lo.y, w_lo.z, w_lo.w, w_hi.x, w_hi.y, w_hi.z, w_hi.w};
#pragma unroll
                    for (int c = 0; c < 8; ++c) dequant_word_bf16(words8[c], scale2, bias2, &wq[4 * c]);
                    if (kb == 0) {
                        if (!ptx::mbar_wait(&stage_empty[group], (use & 1u) ^ 1u, abort_flag, kWaitAbEmpty)) { alive = false; break; }
                        ++use;
                        __syncwarp();  // the .sync.aligned tcgen05 instructions below need a converged warp
                        ptx::tc_fence_after_sync();
                    }
                    if (st * kUmmaKBlocksPerSlot + j < w.nkb) {  // past a ragged end nothing is multiplied
                        ptx::tmem_st16(a_lane + kb * 32, &wq[0]);
                        ptx::tmem_st16(a_lane + kb * 32 + 16, &wq[16]);
                    }
                }
                if (!alive) break;
                ptx::tc_wait_st();
                ptx::tc_fence_before_sync();
                // The ring slot read above with ordinary loads may later be overwritten by TMA (async proxy): order
                // the two.
                ptx::fence_proxy_async_smem();
                __syncwarp();
                if (lane == 0) {
                    ptx::mbar_arrive(&a_full[group]);
                    ptx::mbar_arrive(&ring_empty[at.slot]);
                }
            }
        }
    }

    // ---------------------------------------------------------------------- end; sum over the cluster
    __syncwarp();
    if constexpr (kCluster) {
        const int row_tile = w.first_tile / p.act_tiles;
        const int m_base = (w.first_tile - row_tile * p.act_tiles) * npad, rows = min(npad, p.M - m_base);
        float* staging = p.sum_bytes ? sum_tile : reinterpret_cast<float*>(smem);
        ptx::cluster_wait();
        if (p.sum_bytes == 0) {  // no room beside the rings: over them, when every CTA is done with its own
            ptx::cluster_arrive();
            ptx::cluster_wait();
        }
        if (warp >= kUmmaEpilogueWarp && !*abort_flag)
            umma_push_slices<kSwiglu, kTwo>(p, w, ptx::smem_u32(staging), tmem_base + ((uint32_t)((warp & 3) * 32) << 16), unit_cols, rows,
                                      (warp & 3) * 32 + lane);
        ptx::tc_fence_before_sync();
        __syncwarp();
        ptx::cluster_arrive();
        ptx::cluster_wait();
        umma_finish_rows<kSwiglu>(p, w, staging, m_base, rows, row_tile);
        __syncthreads();
    } else {
        ptx::tc_fence_before_sync();
        __syncthreads();
    }
    if (warp == kUmmaMmaWarp) {
        __syncwarp();
        ptx::tmem_dealloc(tmem_base, kUmmaTmemCols);
    }
}

// ------------------------------------------------------------------------------- host side
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

inline EncodeTiledFn encode_tiled_fn() {
    static EncodeTiledFn fn = []() -> EncodeTiledFn {
        void* ptr = nullptr;
        cudaDriverEntryPointQueryResult result;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &result) != cudaSuccess ||
            result != cudaDriverEntryPointSuccess)
            return nullptr;
        return reinterpret_cast<EncodeTiledFn>(ptr);
    }();
    return fn;
}

// Packed weights as a 2-D uint32 tensor [N, K/8]; box = 32 words (128 B, four k-blocks) x 128 rows,
// 128-byte swizzle so that a thread reading "its" row's 32 bytes hits distinct banks.
// Activations [M, K] as a 3-D bf16 tensor [K/64][M][64]; box = 64 columns (128 B, one k-block) x the padded row
// count x 2 k-blocks, 128-byte swizzle: the box is the B tiles of an activation slot, rows past M read as zero.
// A tensor map is a pure function of (address, extents, box): encoding one costs a microsecond or
// two of host time and a two-kernel MLP needs five, so each host thread remembers the last few it built
// (weights never move, executors reuse their activation buffers).  Direct-mapped, 64 entries.
struct TensorMapKey {
    const void* base;
    int a, b, box_rows, kind;
    bool operator==(const TensorMapKey& o) const {
        return base == o.base && a == o.a && b == o.b && box_rows == o.box_rows && kind == o.kind;
    }
};
struct TensorMapSlot {
    TensorMapKey key;
    CUtensorMap map;
    bool valid;
};
inline TensorMapSlot& tensor_map_slot(const TensorMapKey& key) {
    thread_local TensorMapSlot slots[64] = {};
    const uintptr_t bits = reinterpret_cast<uintptr_t>(key.base) >> 8;
    const size_t index = (size_t)((bits ^ (bits >> 7) ^ (uintptr_t)(key.a * 31 + key.b * 7 + key.box_rows + key.kind * 13)) & 63u);
    return slots[index];
}

inline bool encode_activation_map_uncached(CUtensorMap* map, const void* base, int M, int K, int box_rows) {
    EncodeTiledFn fn = encode_tiled_fn();
    if (!fn) return false;
    cuuint64_t dims[3] = {(cuuint64_t)kUmmaBlockK, (cuuint64_t)M, (cuuint64_t)(K / kUmmaBlockK)};
    cuuint64_t strides[2] = {(cuuint64_t)K * 2, (cuuint64_t)kUmmaBlockK * 2};
    cuuint32_t box[3] = {(cuuint32_t)kUmmaBlockK, (cuuint32_t)box_rows, 2};
    cuuint32_t elem_strides[3] = {1, 1, 1};
    return fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(base), dims, strides, box, elem_strides,
              CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

inline bool encode_weight_map_uncached(CUtensorMap* map, const void* base, int K, int N, int box_rows) {
    EncodeTiledFn fn = encode_tiled_fn();
    if (!fn) return false;
    cuuint64_t dims[2] = {(cuuint64_t)K / 8, (cuuint64_t)N};
    cuuint64_t strides[1] = {(cuuint64_t)K / 2};
    cuuint32_t box[2] = {32, (cuuint32_t)box_rows};
    cuuint32_t elem_strides[2] = {1, 1};
    return fn(map, CU_TENSOR_MAP_DATA_TYPE_UINT32, 2, const_cast<void*>(base), dims, strides, box, elem_strides,
              CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <typename Encode>
inline bool remembered_tensor_map(CUtensorMap* map, const TensorMapKey& key, Encode&& encode) {
    TensorMapSlot& slot = tensor_map_slot(key);
    if (!(slot.valid && slot.key == key)) {
        slot.valid = false;
        if (!encode(&slot.map)) return false;
        slot.key = key;
        slot.valid = true;
    }
    *map = slot.map;
    return true;
}

inline bool encode_activation_map(CUtensorMap* map, const void* base, int M, int K, int box_rows) {
    return remembered_tensor_map(map, TensorMapKey{base, M, K, box_rows, 1},
                                 [&](CUtensorMap* to) { return encode_activation_map_uncached(to, base, M, K, box_rows); });
}

inline bool encode_weight_map(CUtensorMap* map, const void* base, int K, int N, int box_rows = kUmmaTileRows) {
    return remembered_tensor_map(map, TensorMapKey{base, K, N, box_rows, 2},
                                 [&](CUtensorMap* to) { return encode_weight_map_uncached(to, base, K, N, box_rows); });
}

template <bool kSwiglu, bool kCluster, bool kWindows, bool kFew, bool kTwo>
inline cudaError_t configure_umma_instance(int device) {
    static bool configured[64] = {};
    if (device < 64 && configured[device]) return cudaSuccess;
    const cudaError_t rc = cudaFuncSetAttribute(affine_umma_kernel<kSwiglu, kCluster, kWindows, kFew, kTwo>,
                                                cudaFuncAttributeMaxDynamicSharedMemorySize, kUmmaSmemBytes);
    if (rc == cudaSuccess && device < 64) configured[device] = true;
    return rc;
}

// How many clusters of `size` CTAs can be resident at once (size 1: CTAs without a cluster).
template <bool kSwiglu>
inline int umma_active_clusters(int size, int device) {
    static int cached[64][9] = {};
    if (device < 64 && cached[device][size]) return cached[device][size];
    if (configure_umma_instance<kSwiglu, true, false, false, !kSwiglu>(device) != cudaSuccess) return 0;
    cudaLaunchConfig_t config = {};
    config.gridDim = dim3(size * 64, 1, 1);
    config.blockDim = dim3(kUmmaThreads, 1, 1);
    config.dynamicSmemBytes = kUmmaSmemBytes;
    cudaLaunchAttribute attrs[1];
    attrs[0].id = cudaLaunchAttributeClusterDimension;
    attrs[0].val.clusterDim.x = size;
    attrs[0].val.clusterDim.y = 1;
    attrs[0].val.clusterDim.z = 1;
    config.attrs = attrs;
    config.numAttrs = 1;
    int clusters = 0;
    if (cudaOccupancyMaxActiveClusters(&clusters, affine_umma_kernel<kSwiglu, true, false, false, !kSwiglu>, &config) != cudaSuccess) clusters = 0;
    if (device < 64) cached[device][size] = clusters > 0 ? clusters : -1;
    return clusters;
}

// Slices of the K range that are accumulated apart and added in order: part of a result's bits.  Where those may not depend
// on the row count they are a function of (N, K, kernel family, device) only, and how the slices are spread over CTAs
// changes nothing.  The rule: the split over a thread-block cluster that finishes 128-row tiles soonest,
// waves x (k-blocks per CTA + a fixed part).
template <bool kSwiglu>
inline int umma_slices(int N, int slots_total, int device) {
    const int tiles = (N + kUmmaTileRows - 1) / kUmmaTileRows;
    int best = 1;
    long best_cost = -1;
    for (int s = 1; s <= 8; ++s) {
        if (s > slots_total) break;
        const int active = umma_active_clusters<kSwiglu>(s, device);
        if (active <= 0) continue;
        const long waves = (tiles + active - 1) / active;
        const long per_cta = (slots_total + s - 1) / s;
        const long cost = waves * (per_cta * 4 + 6);
        if (best_cost < 0 || cost < best_cost) {
            best_cost = cost;
            best = s;
        }
    }
    return best;
}

// How the work is then laid over the SMs: rows per activation tile and CTAs per tile.  Costs in SM cycles of a B200 at its 1.965 GHz, fitted to measurements of every split at eight shapes and 16 to 512 rows:
//   ring slot (four k-blocks)   530 + 4 per row on a nearly idle chip, 550 + 11 per row with every SM at work (the
//                               activations of all tiles come from L2); never below the weights at 4.8 TB/s
//   CTAs                        45 each, as far as they are resident: what they leave idle, the next kernel starts on
//   finishing a tile            60 per row (40 behind another tile, none where accumulators for both are there)
//   running sum                 14 per row and slice
//   cluster                     45 per row and slice of a CTA; 8000 per wave after the first (it is not persistent)
template <bool kSwiglu>
inline void umma_fixed_plan(UmmaParams& p, int slots_total, int device) {
    p.slices = umma_slices<kSwiglu>(p.N, slots_total, device);
    p.chains = kSwiglu ? 1 : 2;
    long best_cost = -1;
    const int S = p.slices;
    const int splits[3] = {1, (S + 1) / 2, S};
    const long weights = (long)((double)p.N * p.K * (kSwiglu ? 2 : 1) * (0.5625 * 1.965e9 / 4.8e12));
    const int sms = umma_active_clusters<kSwiglu>(1, device);  // with room for a CTA
    if (sms <= 0) return;
    for (int max_rows = kUmmaMaxRows / 2; max_rows <= kUmmaMaxRows; max_rows *= 2) {
        const int act_tiles = (p.M + max_rows - 1) / max_rows;
        const int npad = ((p.M + act_tiles - 1) / act_tiles + 15) / 16 * 16;
        if (max_rows == kUmmaMaxRows && npad <= kUmmaMaxRows / 2) continue;  // the same tiles again
        const bool big = npad > 64;
        const long idle_slot = 530 + 4 * npad, busy_slot = 550 + 11 * npad;
        const long tiles = (long)p.row_tiles * act_tiles;
        for (int i = 0; i < 3; ++i) {
            const int P = splits[i];
            if (i > 0 && P == splits[i - 1]) continue;
            const int active = umma_active_clusters<kSwiglu>(P, device);
            if (active <= 0) continue;
            int local = 0, slots = 0;  // most slices and slots of any CTA of a cluster
            for (int r = 0; r < P; ++r) {
                const int from = S * r / P, to = S * (r + 1) / P;
                const int n = slots_total * to / S - slots_total * from / S;
                local = to - from > local ? to - from : local;
                slots = n > slots ? n : slots;
            }
            const int units = kSwiglu ? (big ? 2 : 4) : (big ? 1 : 2);
            // A cluster's CTA holds its slices, two at most, in units of their own; the running sum over more slices
            // than the final pass reads itself has room for 64 rows.
            if (P > 1 && (local > 2 || local > units)) continue;
            const bool sum = P == 1 && local > (kSwiglu ? 2 : 1);
            if (sum && big) continue;
            const long waves = (tiles + active - 1) / active;
            const long resident = (long)active * P, ctas = tiles * P < resident ? tiles * P : resident;
            const long slot = busy_slot > idle_slot ? idle_slot + (busy_slot - idle_slot) * ctas / sms : idle_slot;
            const long stream = waves * slots * slot;
            long cost = (stream > weights ? stream : weights) + 45 * ctas;
            if (P > 1) {
                cost += 45l * npad * local + (waves - 1) * 8000;
            } else {
                cost += 60l * npad + (units >= 2 * (kSwiglu && local == 2 ? 2 : 1) ? 0 : (waves - 1) * 40l * npad);
                if (sum) cost += waves * (local - 1) * 14l * npad;
            }
            if (best_cost >= 0 && cost >= best_cost) continue;
            best_cost = cost;
            p.act_tiles = act_tiles;
            p.npad = npad;
            p.ksplit = P;
            p.unit_shift = units == 4 ? 2 : units == 2 ? 1 : 0;
            p.sum_bytes = sum ? npad * kUmmaTileRows * 4 : P > 1 && !big ? S * ((npad + P - 1) / P) * kUmmaTileRows * 4 : 0;
        }
    }
}

// Where nothing ties a row's bits to other row counts: a plain projection has one chain too, so that the accumulators of two
// tiles of 128 rows find room and finishing one overlaps the next (in two chains 8192 -> 2048 at 2000 rows took 83 us, now
// 57), and the K range is cut into as many slices as pay for these rows, a CTA each.  Costs in SM cycles at 1.9 GHz, fitted to
// every such split at fourteen shapes and ten row counts from 16 to 2000 in replayed graphs, and to the down projection's in
// eleven MLPs of 9 to 400 rows (what the model picks takes 0.5 and 1.2 % longer than the best split on average, 9 % at most):
//   ring slot (four k-blocks)   923 + 3.2 per row on a nearly idle chip, 12.5 per row with every SM at work; never below the
//                               weights at 4 TB/s
//   CTAs                        3.5 each; 2165 where they find no SMs to start on beside the kernel in front, another like
//                               this one (8192 -> 2048, 16 rows: 64 CTAs 6.6 us, 80 CTAs 7.9) or the MLP's gate|up (1088
//                               / 4096, nine rows, 64 CTAs in front: 72 CTAs 9.6 us, 45 CTAs 10.5)
//   finishing a tile            55 per row, 4 behind another tile
//   cluster                     1180, 64 per row; 8800 + 35 per row for a wave after the first (it is not persistent)
template <bool kSwiglu>
inline void umma_plan(UmmaParams& p, int slots_total, int ctas_before, int device) {
    constexpr int kMostSlices = 8;
    const int sms = umma_active_clusters<kSwiglu>(1, device);  // with room for a CTA
    if (sms <= 0) return;
    const double weights = (double)p.N * p.K * (kSwiglu ? 2 : 1) * (0.5625 / 2120.0);
    double best_cost = -1.0;
    for (int max_rows = kUmmaMaxRows / 2; max_rows <= kUmmaMaxRows; max_rows *= 2) {
        const int act_tiles = (p.M + max_rows - 1) / max_rows;
        const int npad = ((p.M + act_tiles - 1) / act_tiles + 15) / 16 * 16;
        if (max_rows == kUmmaMaxRows && npad <= kUmmaMaxRows / 2) continue;  // the same tiles again
        const long tiles = (long)p.row_tiles * act_tiles;
        const double idle = 923 + 3.2 * npad, busy = 12.5 * npad;
        for (int P = 1; P <= kMostSlices && P <= slots_total; ++P) {
            const int active = umma_active_clusters<kSwiglu>(P, device);
            if (active <= 0) continue;
            const long waves = (tiles + active - 1) / active, ctas = std::min(tiles, (long)active) * P;
            const double slot = busy > idle ? idle + (busy - idle) * ctas / sms : idle;
            double cost = std::max((double)waves * ((slots_total + P - 1) / P) * slot, weights) + 3.5 * ctas;
            if (ctas_before ? ctas_before + ctas > sms : 2 * tiles > active) cost += 2165;
            if (P > 1) cost += 1180 + 64.0 * npad + (waves - 1) * (8800 + 35.0 * npad);
            else cost += 55.0 * npad + (waves - 1) * 4.4 * npad;
            if (best_cost >= 0 && cost >= best_cost) continue;
            best_cost = cost;
            p.act_tiles = act_tiles;
            p.npad = npad;
            p.slices = p.ksplit = P;
            p.chains = 1;
            p.unit_shift = npad > 64 ? 1 : 2;
            p.sum_bytes = P > 1 && npad <= 64 ? P * ((npad + P - 1) / P) * kUmmaTileRows * 4 : 0;
        }
    }
}

template <bool kSwiglu, bool kCluster, bool kWindows, bool kFew, bool kTwo>
inline int launch_umma_instance(const UmmaParams& params, int ctas, int device, cudaStream_t stream) {
    if (configure_umma_instance<kSwiglu, kCluster, kWindows, kFew, kTwo>(device) != cudaSuccess) return MT_ERR_LAUNCH;
    cudaLaunchConfig_t config = {};
    config.gridDim = dim3(ctas, 1, 1);
    config.blockDim = dim3(kUmmaThreads, 1, 1);
    config.dynamicSmemBytes = umma_smem_bytes(params.npad);
    config.stream = stream;
    cudaLaunchAttribute attrs[2];
    attrs[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attrs[0].val.programmaticStreamSerializationAllowed = 1;
    attrs[1].id = cudaLaunchAttributeClusterDimension;
    attrs[1].val.clusterDim.x = params.ksplit;
    attrs[1].val.clusterDim.y = 1;
    attrs[1].val.clusterDim.z = 1;
    config.attrs = attrs;
    config.numAttrs = kCluster ? 2 : 1;
    return cudaLaunchKernelEx(&config, affine_umma_kernel<kSwiglu, kCluster, kWindows, kFew, kTwo>, params) == cudaSuccess ? MT_OK : MT_ERR_LAUNCH;
}

template <bool kSwiglu, bool kWindows, bool kFew, bool kTwo>
inline int launch_umma_tables(const UmmaParams& params, int device, cudaStream_t stream) {
    const int tiles = params.row_tiles * params.act_tiles;
    if (params.ksplit > 1) return launch_umma_instance<kSwiglu, true, kWindows, kFew, kTwo>(params, tiles * params.ksplit, device, stream);
    const int resident = umma_active_clusters<kSwiglu>(1, device);
    return launch_umma_instance<kSwiglu, false, kWindows, kFew, kTwo>(params, tiles < resident ? tiles : resident, device, stream);
}

template <bool kSwiglu, bool kTwo>
inline int launch_umma_chains(const UmmaParams& params, bool windows, int device, cudaStream_t stream) {
    if (windows) return launch_umma_tables<kSwiglu, true, false, kTwo>(params, device, stream);
    return params.npad <= 32 ? launch_umma_tables<kSwiglu, false, true, kTwo>(params, device, stream)
                             : launch_umma_tables<kSwiglu, false, false, kTwo>(params, device, stream);
}

template <bool kSwiglu>
inline int launch_umma_family(UmmaParams& params, bool invariant, int* ctas, cudaStream_t stream) {
    int device = 0;
    if (cudaGetDevice(&device) != cudaSuccess) return MT_ERR_DEVICE;
    const int kblocks = params.K / kUmmaBlockK;
    const int slots_total = (kblocks + kUmmaKBlocksPerSlot - 1) / kUmmaKBlocksPerSlot;
    params.npad = 0;
    if (invariant) umma_fixed_plan<kSwiglu>(params, slots_total, device);
    else umma_plan<kSwiglu>(params, slots_total, ctas ? *ctas : 0, device);
    if (params.npad == 0) return MT_ERR_LAUNCH;  // not even one CTA fits the device
    if (ctas) *ctas = std::min(params.row_tiles * params.act_tiles, umma_active_clusters<kSwiglu>(1, device)) * params.ksplit;
    params.side_bytes = params.sum_bytes + (params.residual && params.ksplit == 1 ? kUmmaResidualBytes : 0);
    if (!encode_activation_map(&params.x_map, params.x, params.M, params.K, params.npad)) return MT_ERR_LAUNCH;
    bool windows = kblocks % 4 != 0;
    for (int t = 0; t < 2; ++t) windows = windows || !aligned_to(params.scales[t], 8) || !aligned_to(params.biases[t], 8);
    if (!kSwiglu && params.chains == 2) return launch_umma_chains<kSwiglu, !kSwiglu>(params, windows, device, stream);
    return launch_umma_chains<kSwiglu, false>(params, windows, device, stream);
}

struct AffineWeights {
    const uint32_t* w;
    const uint16_t* scales;
    const uint16_t* biases;
};

// x [M,K] bf16, one weight triple (plain / residual) or two (gate, up -> SwiGLU).  `invariant`: a row's bits do not depend on M.
// `ctas`, where given: CTAs of the kernel in front (0: unknown) before, of this one after.
inline int launch_umma(const void* x, const AffineWeights* first, const AffineWeights* second, const void* residual,
                       void* out, int M, int K, int N, bool invariant, int* ctas, cudaStream_t stream) {
    if (M < 1 || K % kUmmaBlockK || K < kUmmaBlockK || N < 1) return MT_ERR_SHAPE;
    if (!aligned_to(x, 16) || !aligned_to(first->w, 16) || (second && !aligned_to(second->w, 16))) return MT_ERR_ALIGN;
    const bool swiglu = second != nullptr;
    UmmaParams params;
    params.x = x;
    params.scales[0] = first->scales;
    params.biases[0] = first->biases;
    params.scales[1] = swiglu ? second->scales : first->scales;
    params.biases[1] = swiglu ? second->biases : first->biases;
    params.residual = static_cast<const uint16_t*>(residual);
    params.out = static_cast<uint16_t*>(out);
    params.M = M;
    params.K = K;
    params.N = N;
    params.row_tiles = swiglu ? (N + 63) / 64 : (N + 127) / 128;
    params.wide_out = N % 8 == 0 && aligned_to(out, 16) && (!residual || aligned_to(residual, 16));
    const int box_rows = swiglu ? 64 : 128;
    if (!encode_weight_map(&params.w_map[0], first->w, K, N, box_rows)) return MT_ERR_LAUNCH;
    if (swiglu && !encode_weight_map(&params.w_map[1], second->w, K, N, box_rows)) return MT_ERR_LAUNCH;
    return swiglu ? launch_umma_family<true>(params, invariant, ctas, stream) : launch_umma_family<false>(params, invariant, ctas, stream);
}

}  // namespace mt
