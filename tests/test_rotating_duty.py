"""CPU model of the rotating inversion as the search kernel runs it: warp `it mod warps` inverts
iteration it, after its backward pass of iteration it-1, so that it does not wait for the slowest
warp's forward pass.  Random schedules and stop requests, as in test_pipeline_protocol.py."""
import random

import pytest

import test_pipeline_protocol as model


def warp_program(w, warps, iters, state, stop_at, log):
    it = 0
    while True:
        yield ("point",)
        mine = w == it % warps
        if it == 0 or (it < iters and it < state["stop"]):
            log["produced"].append(it)
            if not mine:
                yield ("arrive", 1 + (it & 1), it)
        if it > 0:
            p = it - 1
            if w != p % warps:
                yield ("sync", 3 + (p & 1), p)
            log["done"].append(p)
            yield ("point",)
            if it >= iters or it >= state["stop"]:
                return
        if mine:
            yield ("sync", 1 + (it & 1), it)
            if it in stop_at:
                yield ("point",)
                state["stop"] = min(state["stop"], it + 2)
            yield ("point",)
            yield ("arrive", 3 + (it & 1), it)
        it += 1


@pytest.mark.parametrize("warps", [8, 16])
@pytest.mark.parametrize("iters", [1, 2, 3, 17, 40])
def test_no_schedule_deadlocks(monkeypatch, warps, iters):
    monkeypatch.setattr(model, "warp_program", warp_program)
    for seed in range(20):
        rng = random.Random(seed)
        stop_at = set(rng.sample(range(iters), rng.randint(0, min(2, iters))))
        length = model.run_schedule(warps, iters, stop_at, rng)
        assert length == min([iters] + [it + 2 for it in stop_at])
