// Rows of a table by index: the token embedding in front of a model's first block.
//
// Bound by latency: a decode step gathers a row per sequence.  The framework's kernel for up to sixteen indices walks the
// elements with a division each (16 rows of 1536: 13.4 us in a replayed graph); here a CTA has a row, its threads 16 bytes
// each, and the launch overlaps its neighbours (1.6 us).
#pragma once

#include "common.cuh"
#include "ptx.cuh"

namespace mt {

constexpr int kGatherThreads = 256;
constexpr unsigned int kGatherIndexOutside = 0x301;

// out[r] = table[index[r]], rows of `vectors` 16-byte vectors; an index outside the table gives a row of NaN and is recorded.
__global__ void __launch_bounds__(kGatherThreads) gather_rows_kernel(const uint4* table, const long long* index, uint4* out, long long table_rows, int vectors) {
    ptx::griddep_launch_dependents();
    ptx::griddep_wait();  // the indices are, and the output may still be read by, a preceding kernel
    long long row;
    asm volatile("ld.global.s64 %0, [%1];" : "=l"(row) : "l"(index + blockIdx.x));
    const bool inside = row >= 0 && row < table_rows;
    if (!inside && threadIdx.x == 0 && atomicCAS(&g_device_status[0], 0u, kGatherIndexOutside) == 0u) {
        g_device_status[1] = blockIdx.x;
        g_device_status[2] = (unsigned int)row;
        g_device_status[3] = (unsigned int)(row >> 32);
    }
    const uint4* from = table + (inside ? row : 0) * (long long)vectors;
    uint4* to = out + (long long)blockIdx.x * vectors;
    for (int i = threadIdx.x; i < vectors; i += blockDim.x) {
        uint4 v = make_uint4(0x7FFF7FFFu, 0x7FFF7FFFu, 0x7FFF7FFFu, 0x7FFF7FFFu);
        if (inside) v = ptx::ld_global_dependent_u4(from + i);
        to[i] = v;
    }
}

inline int launch_gather_rows(const void* table, const long long* index, void* out, int rows, long long table_rows, int width, cudaStream_t stream) {
    if (width % 8 || !aligned_to(table, 16) || !aligned_to(out, 16) || !aligned_to(index, 8)) return MT_ERR_ALIGN;
    cudaLaunchConfig_t config = {};
    const int vectors = width / 8;
    config.gridDim = dim3(rows, 1, 1);
    config.blockDim = dim3(vectors < kGatherThreads ? (vectors + 31) / 32 * 32 : kGatherThreads, 1, 1);
    config.stream = stream;
    cudaLaunchAttribute attrs[1];
    attrs[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attrs[0].val.programmaticStreamSerializationAllowed = 1;
    config.attrs = attrs;
    config.numAttrs = 1;
    return cudaLaunchKernelEx(&config, gather_rows_kernel, static_cast<const uint4*>(table), index, static_cast<uint4*>(out), table_rows, vectors) == cudaSuccess
               ? MT_OK : MT_ERR_LAUNCH;
}

}  // namespace mt
