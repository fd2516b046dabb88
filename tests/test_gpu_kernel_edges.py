"""The edges of the kernels' tiles, chunks and rings, against the CPU oracle or rows run alone."""
import contextlib
import ctypes

import pytest
import torch

from metile_b200 import _lib, backends as B, synth
from metile_b200.backends import cuda_quantized
from metile_b200.integrations import blocks
from oracle import affine as A
from oracle import attention as OA
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


@pytest.mark.parametrize("rows,k,n", [
    (2, 64, 5),           # one k-block
    (16, 8192, 2048),     # four slices over clusters
    (48, 1088, 700),      # slices of unequal length, unaligned tables
    (65, 1536, 1003),     # two tiles of activations, odd rows
    (128, 8960, 1536),    # five slices
    (300, 2048, 2112),    # one slice, tiles of 112 rows
])
def test_tcgen05_sums_cut_for_the_rows_and_for_all(cuda_device, rows, k, n):
    """A call on its own is cut as its rows need; within fixed_order() its bits are batch-invariant mode's."""
    x = synth.activations(1, rows, k, cuda_device)
    triple, other = synth.affine_weight(2, n, k, cuda_device), synth.affine_weight(4, n, k, cuda_device)
    r = synth.activations(3, rows, n, cuda_device)
    calls = [lambda: B.mlx_affine_qmv(x, *triple), lambda: B.mlx_affine_residual_qmv(x, *triple, r),
             lambda: B.mlx_affine_swiglu(x, *triple, *other)]
    own = [call() for call in calls]
    with B.batch_invariant():
        invariant = [call() for call in calls]
    with B.fixed_order():
        fixed = [call() for call in calls]
    assert not B.kernel_pinned()
    for a, b in zip(fixed, invariant):
        assert_bit_equal(a, b, "fixed order")
    weights, up = triple_np(triple), triple_np(other)
    some = sorted({0, rows // 2, rows - 1})
    for outputs in (own, fixed):
        assert_within(outputs[0][some], A.qmm(f32(x[some]), *weights, weights="bf16"))
        assert_within(outputs[1][some], A.qmm(f32(x[some]), *weights, residual=f32(r[some]), weights="bf16"))
        assert_within(outputs[2][some], A.swiglu_fused(f32(x[some]), weights, up, weights="bf16"))


@pytest.mark.parametrize("k,n", [
    (512, 16401),         # one item per row; a last tile of one row, whose tables end within sixteen bytes
    (704, 16001),         # items of eight and of three groups
    (1536, 5500),         # three items over three warps
    (2048, 40000),        # several tiles per team
    (2560, 6007),         # five items over four warps
    (4096, 11100),        # eight items
    (14336, 4840),        # a long K range, beyond the rings of the CUDA-core form
])
def test_one_row_on_warp_mma(cuda_device, k, n):
    """The default form of one row against the CUDA-core form (both keep the weights exact) and the oracle."""
    x, r = synth.activations(1, 1, k, cuda_device), synth.activations(3, 1, n, cuda_device)
    triple, other = synth.affine_weight(2, n, k, cuda_device), synth.affine_weight(4, n, k, cuda_device)
    odd = torch.empty(n + 1, dtype=r.dtype, device=r.device)[1:].view_as(r).copy_(r)
    calls = [lambda: B.mlx_affine_qmv(x, *triple), lambda: B.mlx_affine_residual_qmv(x, *triple, r),
             lambda: B.mlx_affine_swiglu(x, *triple, *other)]
    own = [call() for call in calls]
    for a, b in zip(own, [call() for call in calls]):
        assert_bit_equal(a, b, "twice")
    assert_bit_equal(B.mlx_affine_residual_qmv(x, *triple, odd), own[1], "a residual at an odd address")
    with B.force_kernel("gemv"):
        cores = [call() for call in calls]
    with B.fixed_order():
        for a, b in zip([call() for call in calls], cores):
            assert_bit_equal(a, b, "a model's call")
    # Tables that do not start at sixteen bytes are served by the CUDA-core form.
    shifted = [torch.empty(t.numel() + 1, dtype=t.dtype, device=t.device)[1:].view_as(t).copy_(t) for t in triple[1:]]
    assert_bit_equal(B.mlx_affine_qmv(x, triple[0], *shifted), cores[0], "tables at odd addresses")
    for a, b in zip(own, cores):
        assert_within(a, f32(b), rel=1e-5)  # fp32 sums of the same products in two orders, one rounding each
    weights = triple_np(triple)
    assert_within(own[0], A.qmm(f32(x), *weights))
    assert_within(own[1], A.qmm(f32(x), *weights, residual=f32(r)))
    assert_within(own[2], A.swiglu_fused(f32(x), weights, triple_np(other)))
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


def at_offset(tensor, elements):
    """The same values `elements` elements into an allocation."""
    return torch.empty(tensor.numel() + elements, dtype=tensor.dtype, device=tensor.device)[elements:].view(tensor.shape).copy_(tensor)


@pytest.mark.parametrize("k,n", [
    (64, 3),          # fewer outputs than a half-warp has rows: the register form
    (64, 4), (64, 5),  # one group per row, rows that share a table word, a last word with one group
    (192, 7),         # three groups, a last task that overlaps its neighbour
    (320, 131),       # five groups
    (4160, 1001),     # K parts that begin in the middle of a group
    (9024, 9),        # 141 groups in eight parts
    (13824, 257),     # the longest row whose activations fit beside the rings
    (13888, 257),     # the first that does not
])
def test_one_row_gemv_edges(cuda_device, k, n):
    x = synth.activations(1, 2, k, cuda_device)
    gate, up = synth.affine_weight(2, n, k, cuda_device), synth.affine_weight(3, n, k, cuda_device)
    r = synth.activations(4, 2, n, cuda_device)
    with B.force_kernel("gemv"):
        # Two rows take the register form: the same sums in the same order.
        two = B.mlx_affine_qmv(x, *gate), B.mlx_affine_residual_qmv(x, *gate, r), B.mlx_affine_swiglu(x, *gate, *up)
    one = B.mlx_affine_qmv(x[:1], *gate), B.mlx_affine_residual_qmv(x[:1], *gate, r[:1]), B.mlx_affine_swiglu(x[:1], *gate, *up)
    for found, wanted, what in zip(one, two, ("plain", "residual", "swiglu")):
        assert_bit_equal(found, wanted[:1], what)
    weights = triple_np(gate)
    assert_within(one[0], A.qmm(f32(x[:1]), *weights))
    assert_within(one[1], A.qmm(f32(x[:1]), *weights, residual=f32(r[:1])))
    assert_within(one[2], A.swiglu_fused(f32(x[:1]), weights, triple_np(up)))
    # Tables off a 4-byte boundary (the register form) and off an 8-byte one.
    for offset in (1, 2):
        moved = gate[0], at_offset(gate[1], offset), at_offset(gate[2], offset)
        assert_bit_equal(B.mlx_affine_residual_qmv(x[:1], *moved, r[:1]), one[1], f"tables {offset} elements on")


@pytest.mark.parametrize("k,n", [(64, 5), (192, 130), (448, 257), (1024, 100)])
@pytest.mark.parametrize("rows", [2, 70])
def test_tcgen05_projection_with_tables_anywhere(cuda_device, rows, k, n):
    x, r = synth.activations(1, rows, k, cuda_device), synth.activations(3, rows, n, cuda_device)
    triple = synth.affine_weight(2, n, k, cuda_device)
    wanted = B.mlx_affine_residual_qmv(x, *triple, r), B.mlx_affine_swiglu(x, *triple, *triple)
    for offset in (1, 2, 3, 4):
        moved = triple[0], at_offset(triple[1], offset), at_offset(triple[2], (offset + 2) % 4)
        assert_bit_equal(B.mlx_affine_residual_qmv(x, *moved, r), wanted[0], f"tables {offset} elements on")
        assert_bit_equal(B.mlx_affine_swiglu(x, *moved, *triple), wanted[1], f"gate's tables {offset} elements on")


@pytest.mark.parametrize("batch,kv_heads,group,dim,tokens", [
    (2, 1, 3, 64, 2100),    # 17 splits: one more than are requested at once
    (1, 2, 8, 128, 4096),   # 32 splits: one round of the lanes
    (3, 2, 2, 64, 4225),    # 34 splits, the last one nearly empty
    (2, 1, 4, 128, 8192),   # 64 splits: two rounds
])
def test_attention_merge_edges(cuda_device, batch, kv_heads, group, dim, tokens):
    q = synth.activations(1, batch * kv_heads * group, dim, cuda_device).view(batch, kv_heads * group, 1, dim)
    k, v = (synth.activations(seed, batch * kv_heads * tokens, dim, cuda_device).view(batch, kv_heads, tokens, dim)
            for seed in (2, 3))
    k[:, :, tokens // 3] *= 4  # the maximum lies in one split
    scale = dim ** -0.5
    assert_within(B.mlx_attention_decode(q, k, v, scale=scale), OA.attention_decode(f32(q), f32(k), f32(v), scale))
    for used in (1, 128, 129, 2048, 2049, tokens - 1, tokens):
        lengths = torch.tensor([used] + [max(1, tokens // 2)] * (batch - 1), dtype=torch.int32, device=cuda_device)
        found = B.mlx_attention_decode(q, k, v, scale=scale, lengths=lengths)
        assert_within(found, OA.attention_decode(f32(q), f32(k), f32(v), scale, lengths=lengths.cpu().numpy()), what=f"{used} in use")


@pytest.mark.parametrize("rows,width", [(3, 8184), (2, 8192), (2, 8200), (3, 16384), (2, 32768), (2, 32776), (3, 8193), (2, 1), (5, 31)])
def test_norm_edges(cuda_device, rows, width):
    x, r = synth.activations(1, rows, width, cuda_device), synth.activations(2, rows, width, cuda_device)
    w = synth.norm_weight(3, width, cuda_device)
    total, norm = B.mlx_add_rms_norm(x, r, w, 1e-6)
    o_total, o_norm = A.add_rmsnorm(f32(x), f32(r), f32(w), 1e-6)
    assert (f32(total) == o_total).all()
    assert_within(norm, o_norm, what="add_rmsnorm")
    assert_within(B.mlx_rms_norm(x, w, 1e-6), A.rmsnorm(f32(x), f32(w), 1e-6), what="rmsnorm")
    # Off a 16-byte boundary: element by element, with sums in another order.
    assert_within(B.mlx_rms_norm(at_offset(x, 1), w, 1e-6), A.rmsnorm(f32(x), f32(w), 1e-6), what="unaligned")


def test_what_the_native_calls_do_not_take_the_general_forms_do(cuda_device):
    rows, k, n = 6, 256, 192
    spaced = synth.activations(1, rows, 2 * k, cuda_device)
    x, wide = spaced[:, :k], spaced[:, :k].contiguous()  # rows apart, and dense
    gate, up = synth.affine_weight(2, n, k, cuda_device), synth.affine_weight(3, n, k, cuda_device)
    down = synth.affine_weight(4, k, n, cuda_device)
    r = synth.activations(5, n, rows, cuda_device).t()
    dense, norm = synth.dense_weight(6, n, k, cuda_device), synth.norm_weight(7, k, cuda_device)
    execute = B.mlx_affine_mlp_executor(wide, *gate, *up, *down, None)
    for call in (lambda v, s: B.mlx_affine_qmv(v, *gate), lambda v, s: B.mlx_affine_residual_qmv(v, *gate, s),
                 lambda v, s: B.mlx_affine_swiglu(v, *gate, *up), lambda v, s: execute(v), lambda v, s: execute(v, v),
                 lambda v, s: B.mlx_dense_residual_qmv(v, dense, s), lambda v, s: B.mlx_dense_swiglu(v, dense, dense),
                 lambda v, s: B.mlx_rms_norm(v, norm, 1e-6), lambda v, s: torch.cat(B.mlx_add_rms_norm(v, v, norm, 1e-6))):
        assert_bit_equal(call(x, r), call(wide, r.contiguous()))
        parameter = torch.nn.Parameter(wide, requires_grad=False)  # a subclass of torch.Tensor
        assert_bit_equal(call(parameter, r), call(wide, r.contiguous()))
    # Attention: heads that are not the cache's order, a query of another stride, lengths that are a view.
    q = synth.activations(8, 2 * 64, 4, cuda_device).view(2, 64, 1, 4).permute(0, 3, 2, 1)
    kv = synth.activations(9, 2 * 300 * 2, 64, cuda_device).view(2, 300, 2, 64).transpose(1, 2)
    lengths = torch.tensor([[7, 0], [300, 0]], dtype=torch.int32, device=cuda_device)
    plain = B.mlx_attention_decode(q.contiguous(), kv.contiguous(), kv.contiguous(), scale=0.1, lengths=lengths[:, 0].contiguous())
    assert_bit_equal(B.mlx_attention_decode(q, kv, kv, scale=0.1, lengths=lengths[:, 0].contiguous()), plain)
    # Logits of another type.
    logits, tokens = torch.randn(3, 50, device=cuda_device), torch.zeros(3, 1, dtype=torch.long, device=cuda_device)
    assert torch.equal(B.greedy_token(logits, tokens), logits) and (tokens == logits.argmax(-1, keepdim=True)).all()


@pytest.mark.parametrize("rows,width,vocab", [(1, 8, 1), (16, 1536, 1000), (17, 2056, 7), (700, 512, 300)])
def test_embedding_rows(cuda_device, rows, width, vocab):
    table = synth.activations(1, vocab, width, cuda_device)
    tokens = torch.randint(0, vocab, (rows, 1), device=cuda_device)
    assert_bit_equal(B.embedding(tokens, table), torch.nn.functional.embedding(tokens, table), "rows")
    outside = tokens.clone()
    outside[0], outside[-1] = -1, vocab
    assert _lib.device_status()[0]
    found = B.embedding(outside, table)
    assert found[0].isnan().all() and found[-1].isnan().all()
    if rows > 2:
        assert_bit_equal(found[1:-1], table[tokens[1:-1]], "rows beside one that is not there")
    ok, words = _lib.device_status()
    row, token = words[1], words[2] | words[3] << 32
    assert not ok and words[0] == 0x301 and (row, token) in ((0, 2**64 - 1), (rows - 1, vocab))
    assert _lib.device_status()[0]
    apart = torch.zeros(rows + 1, 4, dtype=torch.int64, device=cuda_device)[:, ::2]
    assert not apart.is_contiguous()
    for other in (tokens.int(), apart, tokens.cpu()):
        assert B.embedding(other, table) is None
    assert B.embedding(tokens, table.float()) is None and B.embedding(tokens[:0], table) is None
    assert B.embedding(tokens, table.clone().requires_grad_()) is None


@pytest.mark.parametrize("change", [
    lambda e: None,
    lambda e: e.register_forward_hook(lambda module, args, out: 2 * out),
    lambda e: setattr(e, "forward", lambda tokens: 3 * torch.nn.functional.embedding(tokens, e.weight)),
    lambda e: setattr(e, "max_norm", 0.5),
    lambda e: e.weight.requires_grad_(),
    lambda e: setattr(e, "weight", torch.nn.Parameter(e.weight.float(), requires_grad=False)),
])
def test_a_model_embeds_as_its_module_does(cuda_device, change):
    from metile_b200.integrations import blocks

    modules = [torch.nn.Embedding.from_pretrained(synth.activations(1, 50, 64, cuda_device), freeze=True) for _ in range(2)]
    for module in modules:  # a look-up with max_norm changes the table
        change(module)
    tokens = torch.randint(0, 50, (3, 4), device=cuda_device)
    found, wanted = blocks._embed(modules[0], tokens), modules[1](tokens)
    assert found.dtype == wanted.dtype and torch.equal(found, wanted) and found.requires_grad == wanted.requires_grad


@pytest.mark.parametrize("family,rows,hidden,inter", [
    ("mlp_fused", 1, 1024, 1024), ("mlp_fused", 1, 2048, 8192), ("mlp_fused", 1, 4096, 2048), ("mlp_fused", 1, 1024, 8192),
    ("mlp_fused", 3, 4096, 8192), ("mlp_fused_mma", 8, 2048, 8192), ("mlp_fused_mma", 2, 512, 1536), ("mlp_fused_mma", 5, 2048, 1024),
])
def test_single_launch_mlp_whose_ctas_do_not_wait(cuda_device, family, rows, hidden, inter):
    """Between the projections a CTA may leave its down rows to the last CTA to arrive, as it does when others are kept off
    the chip.  Without patience nearly all do; whoever sums a row, its bits are the same."""
    gate, up, down = synth.mlp_weights(330, hidden, inter, cuda_device)
    x, res = synth.activations(5, rows, hidden, cuda_device), synth.activations(6, rows, hidden, cuda_device)
    execute = B.mlx_affine_mlp_executor(x, *gate, *up, *down, res)
    state = cuda_quantized._state
    with B.force_kernel(family):
        want = execute(x, res)
        state.flags |= _lib.FLAG_MLP_IMPATIENT
        for _ in range(100):  # more launches than barrier slots
            assert_bit_equal(execute(x, res), want, "rows left to the last CTA")
    assert_within(want, A.mlp(f32(x), *[triple_np(t) for t in (gate, up, down)], f32(res)), rel=3e-3, what="single-launch MLP")
    streams = [torch.cuda.Stream() for _ in range(3)]
    outs = [[] for _ in streams]
    for stream in streams:
        stream.wait_stream(torch.cuda.current_stream())
    executors = [B.mlx_affine_mlp_executor(x, *gate, *up, *down, res) for _ in streams]
    with B.force_kernel(family):
        for _ in range(10):  # side by side: some CTAs find no room while others wait
            for out, stream, run in zip(outs, streams, executors):
                with torch.cuda.stream(stream):
                    out.append(run(x, res))
    torch.cuda.synchronize()
    for out in outs:
        for y in out:
            assert_bit_equal(y, want, "side by side")


@pytest.mark.parametrize("family,rows,hidden,inter", [("mlp_fused", 1, 1024, 1024), ("mlp_fused_mma", 8, 512, 512)])
def test_single_launch_mlps_of_many_streams_meet_apart(cuda_device, family, rows, hidden, inter):
    """Queues of three streams that reach any two launches at once, and more streams than there are meeting slots."""
    gate, up, down = synth.mlp_weights(331, hidden, inter, cuda_device)
    count = 200
    xs = [synth.activations(seed, rows, hidden, cuda_device) for seed in range(count)]
    execute = B.mlx_affine_mlp_executor(xs[0], *gate, *up, *down, None)
    with B.force_kernel(family):
        wanted = [execute(x) for x in xs]
        streams = [torch.cuda.Stream() for _ in range(3)]
        outs = [[] for _ in streams]
        for stream in streams:
            stream.wait_stream(torch.cuda.current_stream())
        for out, stream in zip(outs, streams):
            with torch.cuda.stream(stream):
                torch.cuda._sleep(4_000_000)  # the queues fill up before they begin
                out.extend(execute(x) for x in xs)
        torch.cuda.synchronize()
        for out in outs:
            assert_bit_equal(torch.cat(out), torch.cat(wanted), "side by side")
        # Streams without end: beyond 512 they share a slot, in turn.
        runtime = torch.cuda.cudart()
        handles = (ctypes.c_void_p * 700)()
        outs = []
        for i in range(len(handles)):
            assert int(runtime.cudaStreamCreate(ctypes.addressof(handles) + 8 * i)) == 0
            with torch.cuda.stream(torch.cuda.ExternalStream(handles[i])):
                outs.append(execute(xs[i % count]))
        torch.cuda.synchronize()
        for handle in handles:
            assert int(runtime.cudaStreamDestroy(handle)) == 0
        for i, out in enumerate(outs):
            assert torch.equal(out, wanted[i % count]), i
    assert _lib.device_status()[0]


@pytest.mark.parametrize("batch", [1, 3])
def test_graphs_of_single_launch_mlps_side_by_side(cuda_device, batch):
    """Two decoders of 32 blocks whose captures follow one another launch for launch, replayed on their own streams."""
    from metile_b200.integrations.graphed import GraphedDecoder
    from metile_b200.integrations.torch_lm import apply_metile_to_torch_lm

    model = blocks.random_model(5, hidden=1024, intermediate=1024, heads=4, kv_heads=1, head_dim=64, layers=32, vocab=128,
                                device=cuda_device)
    with apply_metile_to_torch_lm(model, attention=True):
        assert _lib.load().mt_affine_mlp_launches(batch, 1024, 1024, 0) == 1
        prompts = [torch.randint(0, 128, (batch, 9), device=cuda_device, generator=torch.Generator(cuda_device).manual_seed(seed))
                   for seed in (1, 2)]
        tokens = torch.randint(0, 128, (150, batch), device=cuda_device, generator=torch.Generator(cuda_device).manual_seed(3))
        decoders = [GraphedDecoder(model, batch=batch, capacity=200) for _ in prompts]
        wanted = []
        for decoder, prompt in zip(decoders, prompts):
            decoder.prefill(prompt)
            wanted.append([decoder.step(token).clone() for token in tokens])
        torch.cuda.synchronize()
        found = [[], []]
        for decoder in decoders:
            for cache in decoder.cache:
                cache.reset(9)
            decoder.stream.wait_stream(torch.cuda.current_stream())
        for decoder, logits in zip(decoders, found):  # each a queue of its own
            with torch.cuda.stream(decoder.stream):
                torch.cuda._sleep(10_000_000)
        for token in tokens:
            for decoder, logits in zip(decoders, found):
                with torch.cuda.stream(decoder.stream):
                    logits.append(decoder.step(token).clone())
        torch.cuda.synchronize()
    for a, b in zip(found, wanted):
        for x, y in zip(a, b):
            assert torch.equal(x, y)
    assert _lib.device_status()[0]


def opposites(seed, n, k, device):
    """Weights [w, -w], exact in bf16: (q - 8) / 64 with q from 1 to 15, in a triple, and the rms of w."""
    q = torch.randint(1, 16, (n, k // 2), generator=torch.Generator().manual_seed(seed))
    tables = torch.full((n, k // 64), 2.0 ** -6, dtype=torch.bfloat16, device=device)
    return (synth.pack_nibbles(torch.cat([q, 16 - q], dim=1)).to(device), tables, -8 * tables), (q - 8).double().pow(2).mean().sqrt().item() / 64


def error_of_sums(k, codes_from_128=False, peak=1.0):
    """What is left of a sum that is zero is the error of its accumulation, here a share of the sum's size (rms).  A step of a
    tensor-core accumulator (16 products) loses at most 2^-22 of what it holds, sqrt(K / 16) 2^-22 in all.  Where the codes
    are 128 + q, a group's sum is 28 times that of the weights', more where one activation stands out (`peak` times the rms),
    and eight steps lose 28 sqrt(8) 2^-23.  A partial sum of 16 bits would lose 2e-3."""
    return 28 * peak * 8 ** 0.5 * 2 ** -23 if codes_from_128 else (k / 16) ** 0.5 * 2 ** -22


@pytest.mark.parametrize("rows,k,n", [
    (1, 1536, 1536),      # CUDA cores
    (1, 2048, 8192), (1, 4096, 11264),  # warp-level tensor cores
    (2, 1536, 1536), (16, 8192, 2048),  # tcgen05, slices over a cluster
    (128, 8960, 1536), (300, 2048, 2112),
    (2000, 8192, 2048),   # one chain over the whole range
    (100, 27648, 1280),
])
def test_sums_of_projections_are_of_32_bits(cuda_device, rows, k, n):
    weight, size = opposites(1, n, k, cuda_device)
    half = synth.activations(2, rows, k // 2, cuda_device)
    x = torch.cat([half, half], dim=1)
    for order in (contextlib.nullcontext, B.fixed_order, B.batch_invariant):
        with order():
            left = B.mlx_affine_qmv(x, *weight).double()
        cores = rows == 1 and (order is B.fixed_order or (order is contextlib.nullcontext and n * k < 8e6))
        allowed = error_of_sums(k, cores) * size * k ** 0.5
        assert left.pow(2).mean().sqrt().item() <= allowed and left.abs().max().item() <= 8 * allowed, order.__name__


@pytest.mark.parametrize("rows,hidden,inter,codes_from_128", [
    (1, 2048, 8192, False), (1, 1024, 1024, False),  # the single launch of one row
    (8, 2048, 8192, True),                           # and of more
    (1, 4096, 14336, False),                         # two launches on the warp-level tensor cores
    (1, 1536, 8960, True),                           # on the CUDA cores
    (16, 2048, 8192, False), (300, 1536, 8960, False),
])
def test_sums_of_mlps_are_of_32_bits(cuda_device, rows, hidden, inter, codes_from_128):
    """The two halves of the hidden row are the same, those of the down weights opposites."""
    gate, up = ([torch.cat([t, t]) for t in synth.affine_weight(seed, inter // 2, hidden, cuda_device)] for seed in (1, 2))
    down, size = opposites(3, hidden, inter, cuda_device)
    x = synth.activations(4, rows, hidden, cuda_device)
    left = B.mlx_affine_mlp_executor(x, *gate, *up, *down, None)(x).double()
    activations = B.mlx_affine_swiglu(x, *gate, *up).double()
    rms = activations.pow(2).mean().sqrt().item()
    allowed = error_of_sums(inter, codes_from_128, activations.abs().max().item() / rms) * size * rms * inter ** 0.5
    assert left.pow(2).mean().sqrt().item() <= allowed and left.abs().max().item() <= 8 * allowed
