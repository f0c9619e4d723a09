"""Launches whose runs of 8 keys do not fill the threads of a whole iteration: spans counted in 4
and 16 keys per thread, in all or all but one warp of a CTA, one to three iterations."""
import pytest

import meikey_b200 as mk
from conftest import chacha_key

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", params=[(4, 512, 0), (16, 512, 0), (16, 256, 1)], ids=lambda p: "kpt%d-b%d-rot%d" % p)
def runs_ctx(request):
    kpt, block, rot = request.param
    ctx = mk.Context(device=0, table_rows=16, keys_per_thread=kpt, block=block, inverter_rotates=bool(rot),
                     hit_capacity=1 << 18)
    yield ctx
    ctx.close()


@pytest.mark.parametrize("iters", [1, 2, 3])
def test_candidates_of_the_whole_span_and_no_more(runs_ctx, oracle, iters):
    key, base, n = chacha_key(5), 2**35 + 3, runs_ctx.keys_per_iter * iters
    with runs_ctx.job(key, mk.SEED_COUNTER, [mk.Needle.contains("q7x")]) as job:
        job.launch(base, iters)
        hits, total = job.hits(cap=1 << 18)
    want = oracle.search(key, 1, base, n, b"q7x", 3, False, 0)
    assert want and [i for i, _ in hits] == want and total == len(want)
