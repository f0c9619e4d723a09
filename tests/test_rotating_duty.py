"""The rotating inversion's duty over every warp of a CTA (warp `it mod warps` inverts iteration
it), in the CPU model of the search kernel's barrier protocol."""
import random

import pytest

import test_pipeline_protocol as model


@pytest.mark.parametrize("warps", [8, 16])
@pytest.mark.parametrize("iters", [1, 2, 3, 17, 40])
def test_no_schedule_deadlocks(monkeypatch, warps, iters):
    monkeypatch.setattr(model, "inv_warp", lambda it, w: it % w)
    for seed in range(20):
        rng = random.Random(seed)
        stop_at = set(rng.sample(range(iters), rng.randint(0, min(2, iters))))
        length = model.run_schedule(warps, iters, stop_at, rng)
        assert length == min([iters] + [it + 2 for it in stop_at])
