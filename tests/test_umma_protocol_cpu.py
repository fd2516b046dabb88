"""The barrier protocol of the tcgen05 projection as a model that runs on the CPU under random schedules.

The kernel's warps (metile_b200/csrc/affine_umma.cuh) hand slots, operands and sums to one another through
mbarriers, whose waits see only the parity of a phase.  The model has the same roles, waits and arrivals in the
same order; copies land and the tensor pipe works at arbitrary times.  A buffer that is read while it does not
hold what the reader expects, or a state in which nobody can go on, is a fault.  The kernel is not run on a GPU
to find such a fault: there it would be a wrong sum or a stall."""

import random

import pytest

from tests.helpers import host_program


class Barrier:
    def __init__(self, count):
        self.count = self.left = count
        self.phase = 0

    def arrive(self):
        self.left -= 1
        if self.left == 0:
            self.left = self.count
            self.phase += 1

    def passes(self, parity):
        return (self.phase & 1) != parity


class Fault(Exception):
    pass


def expect(found, wanted, what):
    if found != wanted:
        raise Fault(f"{what}: found {found}, expected {wanted}")


class Pipeline:
    """One CTA.  units: accumulator units; slices of a tile's K range; slots: ring slots of a tile; kblocks: its
    k-blocks; reports: groups that report a ring slot as done; accumulators_last: with one unit, the wait for it comes
    after the turn."""

    def __init__(self, *, ring, reports, x_slots, units, slices, slots, kblocks, tiles, accumulators_last=True, warps=2):
        self.__dict__.update(locals())
        self.ring_full = [Barrier(1) for _ in range(ring)]
        self.ring_empty = [Barrier(reports * warps) for _ in range(ring)]
        self.a_full = [Barrier(warps) for _ in range(2)]
        self.stage_empty = [Barrier(1) for _ in range(2)]
        self.x_full = [Barrier(1) for _ in range(x_slots)]
        self.x_empty = [Barrier(1) for _ in range(x_slots)]
        self.turn = [Barrier(1), Barrier(1)]
        self.acc_full = [Barrier(2) for _ in range(units)]
        self.acc_empty = [Barrier(warps) for _ in range(units)]
        self.ring_holds, self.x_holds = [None] * ring, [None] * x_slots
        self.stage_holds = [[None] * warps for _ in range(2)]
        self.acc_holds = [None] * units
        self.tensor_pipe, self.copies = [], []

    def slice_slot(self, s):
        return self.slots * s // self.slices

    # A role yields the (barrier, parity) it waits for, or None where others may get ahead of it.
    def weight_warp(self):
        for count in range(self.tiles * self.slots):
            slot = count % self.ring
            yield self.ring_empty[slot], (count // self.ring) & 1 ^ 1

            def land(slot=slot, count=count):
                self.ring_holds[slot] = count
                self.ring_full[slot].arrive()
            self.ring_holds[slot] = "a copy under way"
            self.copies.append(land)

    def activation_warp(self):
        for use in range(self.tiles * -(-self.kblocks // 2)):
            slot = use % self.x_slots
            yield self.x_empty[slot], (use // self.x_slots) & 1 ^ 1

            def land(slot=slot, use=use):
                self.x_holds[slot] = use
                self.x_full[slot].arrive()
            self.x_holds[slot] = "a copy under way"
            self.copies.append(land)

    def dequant_warp(self, group, warp):
        uses = 0
        for count in range(self.tiles * self.slots):
            slot = count % self.ring
            if count & 1 != group and self.ring % 2 == 0:
                continue
            yield self.ring_full[slot], (count // self.ring) & 1
            if count & 1 != group:
                if self.reports == 2:
                    self.ring_empty[slot].arrive()
                continue
            expect(self.ring_holds[slot], count, "ring slot")
            yield None
            yield self.stage_empty[group], uses & 1 ^ 1
            uses += 1
            expect(self.ring_holds[slot], count, "ring slot")
            self.stage_holds[group][warp] = count
            yield None
            self.a_full[group].arrive()
            self.ring_empty[slot].arrive()

    def mma_warp(self, mine):
        count = q = use = 0
        for _ in range(self.tiles):
            for s in range(self.slices):
                unit, parity = q % self.units, (q // self.units) & 1 ^ 1
                begin, end = self.slice_slot(s), self.slice_slot(s + 1)
                for st in range(begin, end):
                    uses = [use] if self.kblocks - 4 * st <= 2 else [use, use + 1]
                    use += len(uses)
                    if count & 1 == mine:
                        last = self.accumulators_last and self.units == 1
                        if st == begin and not last:
                            yield self.acc_empty[unit], parity
                        for x in uses:
                            yield self.x_full[x % self.x_slots], (x // self.x_slots) & 1
                        yield self.a_full[mine], (count >> 1) & 1
                        if count:
                            yield self.turn[mine], ((count - 1) >> 1) & 1
                        if st == begin and last:
                            yield self.acc_empty[unit], parity
                        self.issue(count, uses, q, unit, st, begin, end)
                        yield None
                    count += 1
                q += 1

    def issue(self, count, uses, q, unit, st, begin, end):
        def multiply():
            for held in self.stage_holds[count & 1]:
                expect(held, count, "operand stage")
            for x in uses:
                expect(self.x_holds[x % self.x_slots], x, "activation slot")
            if st > begin:
                expect(self.acc_holds[unit], (q, st - begin), "accumulators")
            self.acc_holds[unit] = (q, st - begin + 1)
        self.tensor_pipe.append(multiply)
        self.tensor_pipe.append(self.x_empty[uses[0] % self.x_slots].arrive)
        self.turn[count & 1 ^ 1].arrive()
        if len(uses) > 1:
            self.tensor_pipe.append(self.x_empty[uses[1] % self.x_slots].arrive)
        self.tensor_pipe.append(self.stage_empty[count & 1].arrive)
        self.tensor_pipe += [self.acc_full[unit].arrive] * ((st + 2 >= end) + (end - begin == 1))

    def epilogue_warp(self):
        for q in range(self.tiles * self.slices):
            unit, s = q % self.units, q % self.slices
            yield self.acc_full[unit], (q // self.units) & 1
            for _ in range(3):
                expect(self.acc_holds[unit], (q, self.slice_slot(s + 1) - self.slice_slot(s)), "sums")
                yield None
            self.acc_empty[unit].arrive()

    def run(self, seed):
        """None, or what went wrong under this schedule."""
        rng = random.Random(seed)
        roles = [self.weight_warp(), self.activation_warp(), self.mma_warp(0), self.mma_warp(1)]
        roles += [self.dequant_warp(group, warp) for group in range(2) for warp in range(self.warps)]
        roles += [self.epilogue_warp() for _ in range(self.warps)]
        paces = (0.05, 1, 1, 3, 20)
        pace = [rng.choice(paces) for _ in roles] + [rng.choice(paces[1:]) for _ in range(2)]
        waits = [None] * len(roles)
        running = set(range(len(roles)))
        pipe, copy = len(roles), len(roles) + 1
        try:
            while running or self.tensor_pipe or self.copies:
                ready = [i for i in running if waits[i] is None or waits[i][0].passes(waits[i][1])]
                ready += [pipe] * bool(self.tensor_pipe) + [copy] * bool(self.copies)
                if not ready:
                    return "nobody can go on"
                chosen = rng.choices(ready, [pace[i] for i in ready])[0]
                if chosen == pipe:
                    self.tensor_pipe.pop(0)()
                elif chosen == copy:
                    self.copies.pop(rng.randrange(len(self.copies)))()
                else:
                    try:
                        waits[chosen] = next(roles[chosen])
                    except StopIteration:
                        running.discard(chosen)
                if rng.random() < 0.02:
                    pace[rng.randrange(len(roles))] = rng.choice(paces)
        except Fault as fault:
            return str(fault)
        return None


def faults(schedules, **shape):
    return {fault for seed in range(schedules) if (fault := Pipeline(**shape).run(seed))}


@pytest.mark.parametrize("units", [1, 2, 4])
def test_a_slice_waits_until_the_one_before_has_left_its_accumulators(units):
    shape = dict(ring=4, reports=1, x_slots=5, units=units, slices=1, slots=1, kblocks=4, tiles=9)
    assert not faults(200, **shape)
    # Waiting for the accumulators ahead of the turn is what one unit and slices of one slot do not allow.
    assert bool(faults(50, accumulators_last=False, **shape)) == (units == 1)


GEOMETRY = """
#include <cstdio>
#include "affine_umma.cuh"
int main() {
    using namespace mt;
    for (int npad = 16; npad <= kUmmaMaxRows; npad += 16)
        for (int windows = 0; windows < 2; ++windows)
            for (int sums = 0; sums < 2; ++sums)
                for (int residual = 0; residual < 2; ++residual) {
                    if (sums && npad > 64) continue;
                    const int side = sums * 64 * 512 + residual * kUmmaResidualBytes;
                    const int ring = umma_ring_slots(npad, windows, side);
                    std::printf("%d %d %d\\n", ring, umma_slot_reports(ring) / (kUmmaDequantWarps / 2), umma_x_slots(npad, windows, side));
                }
    std::printf("1 %d %d\\n", umma_slot_reports(1) / (kUmmaDequantWarps / 2), umma_x_slots(128, true, 0));  // window tables, one slot per tile
}
"""


@pytest.fixture(scope="module")
def geometries(tmp_path_factory):
    """(ring slots, groups that report a slot, activation slots) of every launch, from the kernel's own header."""
    return sorted(set(host_program(tmp_path_factory.mktemp("geometry"), GEOMETRY)))


def test_every_ring_of_the_kernel_under_every_shape(geometries):
    assert {ring for ring, _, _ in geometries} >= {1, 3, 4}  # odd lengths among them
    rng = random.Random(1)
    for seed in range(600):
        slots = rng.randint(1, 9)
        ring, reports, x_slots = rng.choice(geometries)
        shape = dict(ring=ring, reports=reports, x_slots=x_slots, units=rng.choice((1, 2, 4)),
                     slices=rng.randint(1, min(8, slots)), slots=slots, kblocks=4 * slots - rng.randint(0, 3),
                     tiles=rng.randint(1, 6))
        fault = Pipeline(**shape).run(seed)
        assert fault is None, (fault, shape, seed)


@pytest.mark.parametrize("ring", [1, 3])
def test_in_an_odd_ring_both_groups_report_a_slot(ring):
    shape = dict(ring=ring, x_slots=5, units=2, slices=1, slots=8 if ring > 1 else 1, kblocks=32 if ring > 1 else 3, tiles=6)
    assert not faults(200, reports=2, **shape)
    assert faults(50, reports=1, **shape)  # although both groups wait for every fill
