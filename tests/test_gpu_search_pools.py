"""Contexts that ask for the largest inversion batches: searches keep at least four inversions per CTA
and iteration, and find the oracle's candidates with them."""
import pytest

import meikey_b200 as mk
from conftest import chacha_key
from test_gpu_parity import _start_scalar

pytestmark = pytest.mark.gpu

MADS_MUL, MADS_INVERT = 144, 18 * (30 * 6 + 2 * 72)  # work_per_key's cost of a product and of an inversion


def pools_of(ctx, source):
    """Inversions per CTA and iteration, from the work a key of the search kernel is counted with."""
    threads = ctx.info["block"] - (32 if source == mk.SEED_INCREMENTAL else 0)
    muls, mads = ctx.work_per_key(source)
    return (mads - MADS_MUL * muls) * threads * (16 if source == mk.SEED_INCREMENTAL else 8) / MADS_INVERT


@pytest.mark.parametrize("kpt,block,hw,rot,batch,hashed,incremental", [
    (16, 512, 0, 0, 7680, 4, 4), (16, 512, 0, 1, 8192, 4, 4), (16, 512, 0, 1, 4096, 4, 4), (16, 256, 0, 1, 4096, 4, 4),
    (16, 512, 4, 0, 2816, 4, None), (8, 512, 0, 0, 1280, 4, 6), (8, 512, 0, 0, 256, 16, 30), (4, 256, 0, 0, 64, 32, 32)])
def test_pools(oracle, kpt, block, hw, rot, batch, hashed, incremental):
    with mk.Context(device=0, table_rows=16, keys_per_thread=kpt, block=block, hash_warps=hw, hit_capacity=1 << 18,
                    inverter_rotates=bool(rot), inversion_batch=batch) as ctx:
        assert ctx.info["inversion_batch"] == batch  # as asked, whatever pools come of it
        for source, want in ((mk.SEED_COUNTER, hashed), (mk.SEED_INCREMENTAL, incremental)):
            if want is None:
                continue
            assert pools_of(ctx, source) == pytest.approx(want, rel=1e-9)
            key = _start_scalar(3) if source == mk.SEED_INCREMENTAL else chacha_key(3)
            with ctx.job(key, source, [mk.Needle.suffix("Zq")]) as job:
                job.launch(2**30 + 7, 3)
                hits, _ = job.hits(cap=1 << 18)
            # the start of the second iteration and the end of the last one
            for first in (2**30 + 7 + ctx.keys_per_iter, 2**30 + 7 + 3 * ctx.keys_per_iter - 100000):
                want = oracle.search(key, source, first, 100000, b"Zq", 2, False, 1)
                assert [i for i, _ in hits if first <= i < first + 100000] == want


@pytest.mark.parametrize("kpt,block,hw,rot,says", [(16, 512, 0, 0, 240), (8, 256, 0, 1, 64), (16, 512, 4, 0, 176)])
def test_info_and_pools_without_a_batch(kpt, block, hw, rot, says):
    with mk.Context(device=0, table_rows=16, keys_per_thread=kpt, block=block, hash_warps=hw,
                    inverter_rotates=bool(rot)) as ctx:
        assert ctx.info["inversion_batch"] == says
        assert pools_of(ctx, mk.SEED_COUNTER) == pytest.approx(32, rel=1e-9)
        assert pools_of(ctx, mk.SEED_INCREMENTAL) == pytest.approx(32, rel=1e-9)
