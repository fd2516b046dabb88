"""The edges of the kernels' tiles, chunks and rings, against the CPU oracle or rows run alone."""
import ctypes

import pytest
import torch

from metile_b200 import _lib, backends as B, synth
from metile_b200.integrations import blocks
from oracle import affine as A
from tests.helpers import assert_bit_equal, assert_within, device_library, f32, triple_np

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,k,n", [
    (1, 128, 1),          # fewer outputs than a warp takes, one block
    (3, 384, 5),          # a chunk with an odd row
    (12, 1024, 130),      # ring shorter than the row, a last task that overlaps its neighbour
    (13, 2304, 1001),     # rows past the chunk's
    (16, 16384, 40),      # activations of sixteen rows do not fit
    (17, 512, 300),       # two chunks
    (620, 256, 96),       # two launches
])
def test_dense_rows_edges(cuda_device, rows, k, n):
    x = synth.activations(1, rows, k, cuda_device)
    w, g = (synth.dense_weight(seed, n, k, cuda_device) for seed in (2, 3))
    r = synth.activations(4, rows, n, cuda_device)
    some = sorted({0, rows // 2, rows - 1})
    y = B.mlx_dense_residual_qmv(x, w, r)
    assert (f32(y[some]) == A.dense_rows(f32(x[some]), f32(w), f32(r[some]))).all()
    swi = B.mlx_dense_swiglu(x, g, w)
    alone = torch.cat([B.mlx_dense_swiglu(x[i:i + 1], g, w) for i in some])
    assert_bit_equal(swi[some], alone, "dense swiglu rows alone")
    # Weights that are 8-byte aligned only.
    shifted = torch.empty(n * k + 4, dtype=w.dtype, device=w.device)[4:].view(n, k).copy_(w)
    assert_bit_equal(B.mlx_dense_residual_qmv(x, shifted, r), y, "dense weights off a 16-byte boundary")


@pytest.mark.parametrize("rows,k,n", [
    (2, 64, 5),           # one k-block, narrow rows, unaligned tables
    (17, 8192, 128),      # slices over a thread-block cluster
    (65, 320, 131),       # the first size with one accumulator unit, odd rows
    (128, 6080, 1000),    # unaligned tables over a long range
    (129, 448, 257),      # two activation tiles
    (300, 1024, 1111),    # several tiles per CTA, odd rows that start on either half of a word
    (445, 4096, 2048),    # the running sum over several slices
])
def test_tcgen05_projection_edges(cuda_device, rows, k, n):
    x = synth.activations(1, rows, k, cuda_device)
    triple = synth.affine_weight(2, n, k, cuda_device)
    r = synth.activations(3, rows, n, cuda_device)
    some = sorted({0, 1, rows // 2, rows - 1})
    with B.force_kernel("umma"):
        plain, added = B.mlx_affine_qmv(x, *triple), B.mlx_affine_residual_qmv(x, *triple, r)
        alone = torch.cat([B.mlx_affine_residual_qmv(x[i:i + 1], *triple, r[i:i + 1]) for i in some])
        assert_bit_equal(added[some], alone, "rows alone")
        # The residual and the output apart by half a word.
        shifted = torch.empty(r.numel() + 1, dtype=r.dtype, device=r.device)[1:].view_as(r).copy_(r)
        assert_bit_equal(B.mlx_affine_residual_qmv(x, *triple, shifted), added, "shifted residual")
        swi = B.mlx_affine_swiglu(x, *triple, *triple)
        alone = torch.cat([B.mlx_affine_swiglu(x[i:i + 1], *triple, *triple) for i in some])
        assert_bit_equal(swi[some], alone, "swiglu rows alone")
    weights = triple_np(triple)
    assert_within(plain[some], A.qmm(f32(x[some]), *weights, weights="bf16"))
    assert_within(added[some], A.qmm(f32(x[some]), *weights, residual=f32(r[some]), weights="bf16"))


@pytest.mark.parametrize("rows,k,n", [
    (300, 64, 20480),     # one ring slot per tile, one accumulator unit, four tiles per CTA
    (300, 256, 20480),
    (2000, 192, 3333),    # the same with unaligned tables, narrow rows
    (2000, 512, 5000),    # two slots per tile
])
def test_tcgen05_projection_of_short_rows_over_many_tiles(cuda_device, rows, k, n):
    x = synth.activations(1, rows, k, cuda_device)
    triple = synth.affine_weight(2, n, k, cuda_device)
    r = synth.activations(3, rows, n, cuda_device)
    y, added = B.mlx_affine_qmv(x, *triple), B.mlx_affine_residual_qmv(x, *triple, r)
    few = [(B.mlx_affine_qmv(x[i:i + 48], *triple), B.mlx_affine_residual_qmv(x[i:i + 48], *triple, r[i:i + 48]))
           for i in range(0, rows, 48)]
    assert_bit_equal(y, torch.cat([plain for plain, _ in few]), "rows in batches of 48")
    assert_bit_equal(added, torch.cat([sums for _, sums in few]), "with a residual")
    some = [0, rows // 2, rows - 1]
    assert_within(y[some], A.qmm(f32(x[some]), *triple_np(triple), weights="bf16"))
    assert _lib.device_status()[0]


@pytest.mark.parametrize("batch,steps,first,heads,kv_heads,dim", [
    (1, 1, 0, 1, 1, 2), (2, 7, 3, 3, 1, 20), (1, 130, 0, 6, 2, 64), (3, 33, 40, 4, 4, 128), (1, 2, 30000, 2, 1, 48),
])
def test_rope_kv_prefill_is_the_op_by_op_form(cuda_device, batch, steps, first, heads, kv_heads, dim):
    q, k, v = (synth.activations(seed, batch * steps, width * dim, cuda_device).view(batch, steps, width, dim)
               for seed, width in ((1, heads), (2, kv_heads), (3, kv_heads)))
    theta, positions = 1e6, torch.arange(first, first + steps, device=cuda_device)
    cache = blocks.KVCache(batch, kv_heads, first + steps + 1, dim, cuda_device)
    cache.reset(first)
    rotated, keys, values = cache.rotate_and_fetch(q, k, v, blocks._rope_frequencies(theta, dim, q.device))
    assert_bit_equal(rotated.transpose(1, 2), blocks._rope(q.transpose(1, 2), positions, theta), "queries")
    assert_bit_equal(keys[:, :, first:], blocks._rope(k.transpose(1, 2), positions, theta), "keys")
    assert_bit_equal(values[:, :, first:], v.transpose(1, 2), "values")
    assert not cache.keys[:, :, :first].any() and not cache.keys[:, :, first + steps:].any()
    assert cache.length == first + steps and (cache.positions == first + steps).all()


def test_last_positions_logits_are_those_of_all_positions(cuda_device):
    model = blocks.random_model(3, device=cuda_device)
    tokens = torch.arange(23, device=cuda_device).view(1, 23)
    with torch.no_grad():
        every, last = model(tokens), model(tokens, logits_to_keep=1)
    assert_bit_equal(last, every[:, -1:], "logits of the last position")


@pytest.mark.parametrize("rows,vocabulary", [(1, 1), (3, 7), (16, 32768), (2, 2047), (5, 40000)])
def test_greedy_token_is_float_and_argmax(cuda_device, rows, vocabulary):
    logits = synth.activations(1, rows, vocabulary, cuda_device).round()   # many equal values
    tokens = torch.full((rows, 1), -1, dtype=torch.long, device=cuda_device)
    for special in (None, float("inf"), float("nan")):
        if special is not None:
            logits[rows // 2, vocabulary // 3:] = special
        assert_bit_equal(B.greedy_token(logits, tokens), logits.float(), "logits")
        assert (tokens == logits.float().argmax(-1, keepdim=True)).all()
    logits[:] = float("-inf")
    B.greedy_token(logits, tokens)
    assert (tokens == logits.float().argmax(-1, keepdim=True)).all()


@pytest.mark.parametrize("batch,heads,kv_heads,dim", [(1, 1, 1, 2), (3, 5, 5, 128), (2, 40, 8, 128)])
def test_rope_append_advances_every_position_once(cuda_device, batch, heads, kv_heads, dim):
    q, k, v = (synth.activations(seed, batch * width, dim, cuda_device).view(batch, width, dim)
               for seed, width in ((1, heads), (2, kv_heads), (3, kv_heads)))
    positions = torch.arange(batch, dtype=torch.int32, device=cuda_device)
    caches = [torch.zeros(batch, kv_heads, batch + 1, dim, dtype=torch.bfloat16, device=cuda_device) for _ in range(4)]
    kept = B.rope_kv_append(q, k, v, positions, *caches[:2], theta=1e4)
    assert (positions.cpu() == torch.arange(batch)).all()
    assert_bit_equal(B.rope_kv_append(q, k, v, positions, *caches[2:], theta=1e4, advance=True), kept, "queries")
    assert (positions.cpu() == torch.arange(batch) + 1).all()
    assert_bit_equal(caches[2], caches[0], "keys")
    assert_bit_equal(caches[3], caches[1], "values")


SWIGLU_SOURCE = """
#include "common.cuh"
// Eight gates per thread: neighbours, or (apart) an eighth of all numbers from one another.
__global__ void compare(unsigned long long* different, unsigned int* example, int apart, float up_value) {
    const unsigned int thread = blockIdx.x * blockDim.x + threadIdx.x;
    float gate[8], up[8], out[8];
    for (int i = 0; i < 8; ++i) {
        gate[i] = __uint_as_float(apart ? thread + ((unsigned int)i << 29) : 8 * thread + i);
        up[i] = up_value;
    }
    mt::swiglu8_f32(gate, up, out);
    for (int i = 0; i < 8; ++i) {
        const float one = mt::swiglu_f32(gate[i], up[i]);
        if (__float_as_uint(one) != __float_as_uint(out[i]) && !(one != one && out[i] != out[i])) {
            atomicAdd(different, 1ull);
            *example = __float_as_uint(gate[i]);
        }
    }
}
extern "C" int run(void* different, void* example, int apart, float up, void* stream) {
    compare<<<1 << 21, 256, 0, (cudaStream_t)stream>>>((unsigned long long*)different, (unsigned int*)example, apart, up);
    return (int)cudaGetLastError();
}
"""


def test_eight_swiglus_have_the_bits_of_one_for_every_gate(cuda_device, tmp_path):
    run = device_library(tmp_path, SWIGLU_SOURCE).run
    counts = torch.zeros(2, dtype=torch.int64, device=cuda_device)
    stream = ctypes.c_void_p(torch.cuda.current_stream(cuda_device).cuda_stream)
    for apart in (0, 1):
        for up in (1.0, -0.37):
            assert run(ctypes.c_void_p(counts.data_ptr()), ctypes.c_void_p(counts[1:].data_ptr()), apart, ctypes.c_float(up),
                       stream) == 0
            assert counts[0].item() == 0, hex(counts[1].item())
