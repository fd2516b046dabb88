"""Index arithmetic of the INT4 projections, restated on the CPU.

The GEMV kernel (metile_b200/csrc/affine_gemv.cuh) hands row blocks blockIdx, blockIdx + grid, ... to a
CTA and lets it run `(row_blocks - 1 - blockIdx) / grid + 1` passes, in unsigned arithmetic.  That
is only right while the grid has at most `row_blocks` CTAs, which the launcher guarantees by
construction; these checks pin both halves for the shapes the library is used with."""

import pytest

from tests.helpers import host_program

SM_COUNT = 148
WARPS = 8


def ksplit_of(k, n):
    ksplit, slots = 1, k >> 5
    while ksplit < 8 and n * ksplit < 16384 and slots // (ksplit * 2) >= 16:
        ksplit *= 2
    return ksplit


def rows_per_half_warp(rows, dual):
    if dual:
        return 2 if rows <= 2 else 1
    return 4 if rows <= 2 else (2 if rows <= 4 else 1)


def launch_geometry(rows, dual, k, n, staged_bytes):
    ksplit = ksplit_of(k, n)
    rows_per_cta = (WARPS // ksplit) * 2 * rows_per_half_warp(rows, dual)
    row_blocks = -(-n // rows_per_cta)
    cap = SM_COUNT * (3 if rows == 1 and staged_bytes <= 72 * 1024 else 2)
    return rows_per_cta, row_blocks, min(row_blocks, cap)


SHAPES = [(1536, 8960), (8960, 1536), (2048, 8192), (8192, 2048), (2048, 128256), (5120, 27648),
          (27648, 5120), (5120, 3456), (3456, 5120), (1536, 256), (64, 64), (4096, 1000)]


@pytest.mark.parametrize("k,n", SHAPES)
@pytest.mark.parametrize("rows", [1, 2, 4, 8])
@pytest.mark.parametrize("dual", [False, True])
def test_every_row_block_runs_exactly_once(k, n, rows, dual):
    staged = k * 4 + (k >> 5) * 4 if rows == 1 else rows * k * 2
    rows_per_cta, row_blocks, grid = launch_geometry(rows, dual, k, n, staged)
    assert 1 <= grid <= row_blocks
    seen = [0] * row_blocks
    for cta in range(grid):
        passes = ((row_blocks - 1 - cta) & 0xFFFFFFFF) // grid + 1
        assert passes >= 1
        for p in range(passes):
            block = p * grid + cta
            assert block < row_blocks  # a pass never starts at or beyond the last row
            seen[block] += 1
    assert seen == [1] * row_blocks
    assert (row_blocks - 1) * rows_per_cta < n <= row_blocks * rows_per_cta


def test_pass_counts_differ_by_at_most_one():
    # N = 8192 with 16-row CTAs: 512 row blocks over 444 CTAs -- 68 CTAs run two passes, the rest one
    # (every CTA used to run two, most of them on rows past the end).
    rows_per_cta, row_blocks, grid = launch_geometry(1, True, 2048, 8192, 2048 * 4 + 256)
    assert (rows_per_cta, row_blocks, grid) == (16, 512, 444)
    passes = [(row_blocks - 1 - cta) // grid + 1 for cta in range(grid)]
    assert passes.count(2) == 68 and passes.count(1) == 376


# ---- one activation row: the ring form of the GEMV ----------------------------------------------------------


def ring_parts(k, n):
    """(first slot, slots' end) of each K part of a row; a slot is 32 columns."""
    ksplit, slots = ksplit_of(k, n), k // 32
    per_part = -(-slots // ksplit)
    return [(part * per_part, min((part + 1) * per_part, slots)) for part in range(ksplit)]


def ring_table_words(entry, slot_begin, slot_end, steps):
    """(step, table word, first byte, bytes) of a row's copies; `entry` is its first group of the part in the array."""
    group_begin, group_end = slot_begin // 2, (slot_end + 1) // 2
    for step in range(steps):
        for word in range(4):
            left = group_end - group_begin + entry % 2 - 2 * word - 8 * step
            at = (entry // 2 + word) * 4 + 16 * step
            if left > 0:
                yield step, word, at, 4 if left > 1 else 2
            if word == 0 and (entry | slot_begin) & 1 and left > 8:
                yield step, 4, at + 16, 4 if left > 9 else 2


RING_SHAPES = [(64, 4), (64, 5), (192, 7), (320, 131), (4160, 1001), (9024, 9), (1536, 8960), (13824, 257), (8192, 130)]


@pytest.mark.parametrize("k,n", RING_SHAPES)
def test_ring_copies_every_scale_and_nothing_outside_the_array(k, n):
    groups, end = k // 64, 2 * n * (k // 64)
    for slot_begin, slot_end in ring_parts(k, n):
        steps = -(-(-(-(k // 32) // len(ring_parts(k, n)))) // 16)
        for row in sorted({0, 1, n // 2, n - 2, n - 1}):
            entry = row * groups + slot_begin // 2
            copied = set()
            for step, word, at, size in ring_table_words(entry, slot_begin, slot_end, steps):
                assert at % 4 == 0 and 0 <= at and at + size <= end
                copied |= {(step, 2 * word + half) for half in range(size // 2)}
            for slot in range(slot_begin, slot_end):
                step, lane = (slot - slot_begin) // 16, (slot - slot_begin) % 16
                half = (slot_begin + lane) // 2 - slot_begin // 2 + entry % 2
                assert (step, half) in copied
                # The half-word read there is the slot's own group.
                assert 2 * (entry // 2) + 8 * step + half == row * groups + slot // 2


@pytest.mark.parametrize("k,n", RING_SHAPES)
@pytest.mark.parametrize("dual", [False, True])
def test_ring_tasks_store_every_row_once(k, n, dual):
    rows, ksplit = 2 if dual else 4, ksplit_of(k, n)
    tasks = -(-n // (2 * rows))
    teams = WARPS // ksplit
    grid = min(-(-n // (teams * 2 * rows)), 2 * SM_COUNT)
    stored = [0] * n
    for cta in range(grid):
        for task0 in range(cta, tasks, teams * grid):  # the same passes for all warps of a CTA
            for team in range(teams):
                task = task0 + team * grid
                for half in range(2):
                    row = min(task * 2 * rows + half * rows, n - rows)
                    for r in range(rows):
                        if task < tasks and row + r >= task * 2 * rows + half * rows:
                            stored[row + r] += 1
    assert stored == [1] * n


# ---- the tables of the tcgen05 projection --------------------------------------------------------------------


def window_copies(start, entries):
    """(window, first byte) of a row's 8-byte table copies; `start` is the byte address of its first entry.  Window 0 is
    the one the row starts in the middle of; window st + 1 belongs to slot st, as does window st of an aligned row."""
    offset = start // 2 % 4
    base = start - 2 * offset
    if offset:
        yield 0, base
    for st in range(-(-entries // 4)):
        left = entries - 4 * st
        there = left - 4 + offset if offset else left
        if there > 0:
            yield st + (offset > 0), base + 8 * (st + (offset > 0))


@pytest.mark.parametrize("groups", [1, 2, 3, 4, 5, 7, 8, 21, 95])
@pytest.mark.parametrize("rows", [1, 2, 3, 4, 129, 130, 131])
@pytest.mark.parametrize("shift", [0, 2, 4, 6])
def test_window_copies_bring_every_entry_and_stay_within_the_arrays_own_windows(groups, rows, shift):
    for row in range(rows):
        start = 1024 + shift + 2 * row * groups
        brought = set()
        for _, at in window_copies(start, groups):
            first, last = 1024 + shift, 1024 + shift + 2 * rows * groups - 2
            assert at % 8 == 0 and first // 8 <= at // 8 <= last // 8
            brought |= set(range(at, at + 8, 2))
        assert brought >= {start + 2 * entry for entry in range(groups)}


@pytest.mark.parametrize("rows,n", [(1, 1), (1, 129), (3, 5), (16, 257), (17, 131), (4, 128)])
@pytest.mark.parametrize("odd", [0, 1])  # the residual starts in the middle of a word
def test_residual_words_bring_every_element_and_stay_within_the_arrays_own_words(rows, n, odd):
    brought = set()
    for m in range(rows):
        start = (odd + m * n) % 2
        for tile in range(0, n, 128):
            for word in range(65 if (odd + m * n + tile) % 2 else 64):
                first = tile + 2 * word - start                     # elements first, first + 1
                if first < n:
                    at = 2 * (odd + m * n + first)
                    assert at % 4 == 0 and 2 * odd // 4 <= at // 4 <= 2 * (odd + rows * n - 1) // 4
                    brought |= {at, at + 2}
    assert brought >= {2 * (odd + i) for i in range(rows * n)}


ONE_ROW_FORM = """
#include <cstdio>
#include "affine_gemv_mma.cuh"
using namespace mt;
int main() {
    const int shapes[][3] = {SHAPES};
    uint16_t* const table = reinterpret_cast<uint16_t*>(64);
    const GemvWeights w{nullptr, table, table}, odd{nullptr, table, table + 1};
    for (const auto& s : shapes) {
        OneRowPlan plan = {};
        const bool serves = one_row_applicable(w, w, s[0], s[1], s[2]) && one_row_plan(plan, s[0], s[1], s[2], 148);
        printf("%d %d\\n", serves && one_row_pays(plan, s[0], s[1], s[2], 148), one_row_applicable(w, odd, s[0], s[1], s[2]));
    }
    return 0;
}
"""


def test_one_row_takes_the_tensor_cores_only_where_the_rings_are_slower(tmp_path):
    """Shapes measured on both sides: (K, N, two matrices) and whether the warp-level tensor cores were faster."""
    faster = {(2048, 128256, 0): 1, (1536, 32768, 0): 1, (1536, 5500, 0): 1, (4096, 14336, 0): 1, (1088, 7424, 0): 1,
              (2048, 8192, 1): 1, (5120, 27648, 1): 1, (4096, 14336, 1): 1, (1536, 8960, 1): 1, (4288, 3959, 1): 1,
              (2048, 4096, 0): 0, (2048, 4805, 0): 0, (13632, 5056, 0): 0, (2048, 157, 0): 0, (4096, 4096, 0): 0,
              (7104, 1312, 1): 0, (12928, 775, 1): 0, (3520, 2688, 1): 0, (3136, 4032, 1): 0, (7232, 1920, 1): 0,
              (10240, 5120, 1): 0, (9344, 4829, 1): 0, (832, 19255, 1): 0, (768, 24293, 1): 0, (1152, 21002, 1): 0}
    rows = host_program(tmp_path, ONE_ROW_FORM.replace("SHAPES", ", ".join("{%d, %d, %d}" % shape for shape in faster)))
    assert dict(zip(faster, (row[0] for row in rows))) == faster
    assert not any(row[1] for row in rows)  # tables that bulk copies do not take
