"""The field inversion by division steps (csrc/modinv.cuh) against Python integers."""
import os
import random
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
P = 2**255 - 19


@pytest.fixture(scope="module")
def binary(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("modinv") / "modinv_check")
    subprocess.run(["g++", "-O2", "-std=c++17", "-o", out, os.path.join(HERE, "c", "modinv_check.cpp")], check=True)
    return out


def values(kind):
    rng = random.Random(3)
    if kind == "edges":  # every 256-bit word pattern the kernels may hand over, not only canonical ones
        near = [0, P, 2 * P, 2**256 - 1, 2**255, 2**254, (P + 1) // 2, 2**30, 2**60, 2**240]
        return sorted({x for n in near for d in range(-3, 4) if 0 <= (x := n + d) < 2**256})
    if kind == "powers":
        return [1 << k for k in range(256)] + [(1 << k) - 1 for k in range(1, 257)]
    if kind == "small":
        return list(range(1, 600)) + [P - k for k in range(1, 600)]
    return [rng.getrandbits(256) for _ in range(4000)]


@pytest.mark.parametrize("kind", ["edges", "powers", "small", "random"])
def test_inverse_matches_python(binary, kind):
    xs = values(kind)
    text = "\n".join(f"{x:064x}" for x in xs)
    got = subprocess.run([binary], input=text, capture_output=True, text=True, check=True).stdout.split()
    assert len(got) == len(xs)
    for x, g in zip(xs, got):
        v = int(g, 16)
        assert v < 2**256 and v % P == (pow(x, -1, P) if x % P else 0), hex(x)
