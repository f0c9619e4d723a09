"""CPU model of the search kernel's loop (csrc/kernels.cu, k_search) in both its forms, with its accesses
to the two product buffers and the one inversion scratch buffer.  Rotating: warp `it mod warps` inverts
iteration it, after its backward pass of iteration it-1.  Dedicated: the last warp only inverts.  Random
schedules and stop requests; two inversions at a time, a product overwritten while it is needed or an
inverse read before it is there fail."""
import random

import pytest

from test_pipeline_protocol import run_programs


class Memory:
    def __init__(self, compute_warps):
        self.prod = [[None] * compute_warps for _ in range(2)]
        self.scratch = None  # the iteration being inverted

    def write(self, w, it):
        assert self.scratch is None or self.scratch % 2 != it % 2, "product written into a buffer being inverted"
        assert self.prod[it & 1][w] in (None, ("used", it - 2)), "inverse overwritten before it was used"
        self.prod[it & 1][w] = ("product", it)

    def use(self, w, it):
        assert self.prod[it & 1][w] == ("inverse", it), "inverse read before it was there"
        self.prod[it & 1][w] = ("used", it)

    def invert(self, it, early=False):
        """The inverting warp between its two barrier operations; `early` arrives before the work is done."""
        if early:
            yield ("arrive", 3 + (it & 1), it)
        assert self.scratch is None, "two inversions share the scratch buffer"
        self.scratch = it
        for w in range(len(self.prod[it & 1])):
            yield ("point",)
            assert self.prod[it & 1][w] == ("product", it), "inverted before every product was there"
            self.prod[it & 1][w] = ("inverse", it)
        self.scratch = None
        if not early:
            yield ("arrive", 3 + (it & 1), it)


def inversion(mem, it, iters, state, stop_at, early):
    yield ("sync", 1 + (it & 1), it)
    if it in stop_at and it + 2 < state["stop"]:
        yield ("point",)
        state["stop"] = it + 2
    yield from mem.invert(it, early)


def inverter(mem, iters, state, stop_at, early):
    it = 0
    while True:
        yield from inversion(mem, it, iters, state, stop_at, early)
        if it + 1 >= iters or it + 1 >= state["stop"]:
            return
        it += 1


def compute(w, duty, mem, iters, state, stop_at, early, done):
    """`duty(it)`: whether warp w inverts iteration it."""
    it = 0
    while True:
        yield ("point",)
        if it == 0 or (it < iters and it < state["stop"]):
            mem.write(w, it)
            if not duty(it):
                yield ("arrive", 1 + (it & 1), it)
        if it > 0:
            if not duty(it - 1):
                yield ("sync", 3 + (it - 1 & 1), it - 1)
            mem.use(w, it - 1)
            done.append(it - 1)
            yield ("point",)
            if it >= iters or it >= state["stop"]:
                return
        if duty(it):
            yield from inversion(mem, it, iters, state, stop_at, early)
        it += 1


def run(warps, iters, stop_at, rng, rotating, early=False):
    n = warps if rotating else warps - 1
    mem, state, done = Memory(n), {"stop": iters}, [[] for _ in range(n)]
    progs = [compute(w, (lambda it, w=w: rotating and w == it % warps), mem, iters, state, stop_at, early, done[w])
             for w in range(n)]
    if not rotating:
        progs.append(inverter(mem, iters, state, stop_at, early))
    run_programs(progs, {k: warps for k in (1, 2, 3, 4)}, rng)
    assert done == [list(range(min([iters] + [it + 2 for it in stop_at])))] * n


@pytest.mark.parametrize("rotating", [True, False], ids=["rotating", "dedicated"])
@pytest.mark.parametrize("warps", [8, 16])
def test_buffers(warps, rotating):
    rng = random.Random(warps)
    for _ in range(60):
        iters = rng.choice([1, 2, 3, 4, 5, 9, 20])
        run(warps, iters, set(rng.sample(range(iters), rng.randint(0, min(2, iters)))), rng, rotating)


@pytest.mark.parametrize("rotating", [True, False], ids=["rotating", "dedicated"])
def test_the_model_sees_an_early_arrival(rotating):
    with pytest.raises(AssertionError):
        for seed in range(200):
            run(8, 9, set(), random.Random(seed), rotating, early=True)
