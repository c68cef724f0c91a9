"""Slots of K and V tiles of the two-tile prefill attention, over orders in which its warps can run.

The kernel's two producers, two issuers and two softmax warpgroups, the copies and the tensor core's products are stepped in random
order, with barriers that know what the hardware's know: the parity of a phase.  No schedule may multiply a tile that is not there or
copy over one that is still to be multiplied.
"""
import random
import re
from collections import deque
from pathlib import Path

import pytest

SOURCE = Path(__file__).resolve().parent.parent / "sglang.cpp_b200" / "csrc" / "attention_prefill_tc2.cu"


class Barrier:
    def __init__(self, arrivals=1):
        self.arrivals = self.pending = arrivals
        self.phase = 0                      # the one that is running

    def arrive(self):
        self.pending -= 1
        if self.pending == 0:
            self.pending, self.phase = self.arrivals, self.phase + 1

    def over(self, parity):
        return (self.phase & 1) != parity


class Fault(Exception):
    pass


class Run:
    """``place(kind, kt)``: the slot of a tile and the parity of its use there."""

    def __init__(self, slots, place, tiles, rng):
        self.place, self.tiles, self.rng = place, tiles, rng
        self.full = [Barrier() for _ in range(slots)]
        self.empty = [Barrier() for _ in range(slots)]
        self.holds = [None] * slots         # (kind, kt, products that will still read it)
        self.copies, self.products = [], deque()
        self.s_full, self.s_free, self.p_full, self.pv_done = ([Barrier() for _ in range(2)] for _ in range(4))

    def producer(self, kind):
        for kt in range(self.tiles):
            slot, use = self.place(kind, kt)
            yield lambda: self.empty[slot].over(use ^ 1)
            if self.holds[slot] is not None and self.holds[slot][2] > 0:
                raise Fault(f"{kind}{kt} copied over {self.holds[slot]}")
            self.holds[slot] = [kind, kt, 2]
            self.copies.append((slot, kind, kt))

    def multiply(self, kind, kt, done):
        slot, _ = self.place(kind, kt)
        self.products.append((slot, kind, kt, done))

    def issuer(self, kind):
        for kt in range(self.tiles):
            slot, use = self.place(kind, kt)
            yield lambda: self.full[slot].over(use)
            for i in range(2):
                if kind == "K":
                    if i == 1 or kt > 0:
                        yield lambda: self.s_free[i ^ 1].over((kt & 1) if i == 1 else (kt & 1) ^ 1)
                    done = [self.s_full[0]] if i == 0 else [self.s_full[1], self.empty[slot]]
                else:
                    yield lambda: self.p_full[i].over(kt & 1)
                    done = [self.pv_done[0]] if i == 0 else [self.pv_done[1], self.empty[slot]]
                self.multiply(kind, kt, done)

    def softmax(self, i):
        for kt in range(self.tiles):
            yield lambda: self.s_full[i].over(kt & 1)
            self.s_free[i].arrive()
            if kt > 0:
                yield lambda: self.pv_done[i].over((kt - 1) & 1)
            self.p_full[i].arrive()
        yield lambda: self.pv_done[i].over((self.tiles - 1) & 1)

    def copy_lands(self):
        while True:
            yield lambda: self.copies
            slot, kind, kt = self.copies.pop(self.rng.randrange(len(self.copies)))
            self.landed = getattr(self, "landed", set()) | {(kind, kt)}
            self.full[slot].arrive()

    def product_ends(self):
        while True:
            yield lambda: self.products
            slot, kind, kt, done = self.products.popleft()
            here = self.holds[slot]
            if here is None or here[:2] != [kind, kt] or (kind, kt) not in self.landed:
                raise Fault(f"product of {kind}{kt} read {here}")
            here[2] -= 1
            for b in done:
                b.arrive()

    def walk(self):
        actors = [self.producer("K"), self.producer("V"), self.issuer("K"), self.issuer("V"), self.softmax(0), self.softmax(1)]
        units = [self.copy_lands(), self.product_ends()]
        speed = {id(a): self.rng.choice([0.02, 0.2, 1.0]) for a in actors + units}   # some far behind the others
        waits = {id(a): next(a) for a in actors + units}
        live, idle = set(map(id, actors)), 0
        while live:
            if idle > 10000:
                raise Fault("nobody can go on")
            idle += 1
            for a in actors + units:
                if id(a) not in waits or self.rng.random() > speed[id(a)] or not waits[id(a)]():
                    continue
                idle = 0
                try:
                    waits[id(a)] = a.send(None)
                except StopIteration:
                    live.discard(id(a))
                    del waits[id(a)]


def ring_per_kind(k_slots, v_slots):
    def place(kind, kt):
        n, first = (k_slots, 0) if kind == "K" else (v_slots, k_slots)
        return first + kt % n, kt // n & 1
    return k_slots + v_slots, place


def one_ring(slots):
    def place(kind, kt):
        item = 2 * kt + (kind == "V")
        return item % slots, item // slots & 1
    return slots, place


def kernels_rings():
    source = SOURCE.read_text()
    m = re.search(r"kKSlots = (\d+), kVSlots = (\d+)", source)
    if m:
        return ring_per_kind(int(m[1]), int(m[2]))
    return one_ring(int(re.search(r"constexpr int kSlots = (\d+);", source)[1]))


def walks(rings, count):
    for seed in range(count):
        rng = random.Random(seed)
        Run(*rings, tiles=rng.choice([1, 2, 3, 5, 8, 13]), rng=rng).walk()


def test_every_tile_is_multiplied_where_it_was_copied_to():
    walks(kernels_rings(), 1500)


def test_tiles_of_both_kinds_in_turn_through_one_ring_of_five_are_caught():
    """(each slot holds tiles of both kinds: a parity is that of the phase two before, for all that its tester knows)"""
    with pytest.raises(Fault):
        walks(one_ring(5), 1500)
