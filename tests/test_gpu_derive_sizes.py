"""mk_derive at the sizes where its keys per thread change (1, 2, 4, 8, 16 for up to one wave of 512
threads per SM each) and around them, against the oracle at both ends and across the middle."""
import pytest

import meikey_b200 as mk
from conftest import chacha_key
from test_gpu_parity import _start_scalar

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("source", [mk.SEED_CHACHA20, mk.SEED_COUNTER, mk.SEED_INCREMENTAL])
@pytest.mark.parametrize("waves,off", [(0, 1), (0, 33), (1, 0), (1, 1), (2, 1), (4, -1), (4, 1), (8, 1), (16, 1)])
def test_keys_at_the_edges_of_a_wave(gpu_ctx, oracle, source, waves, off):
    n = waves * gpu_ctx.info["sms"] * 512 + off
    key = _start_scalar(9) if source == mk.SEED_INCREMENTAL else chacha_key(9)
    first = 2**33 + 5
    got = gpu_ctx.derive(key, source, first, n)
    assert len(got) == 32 * n
    for a in {0, n // 2, max(0, n - 70)}:
        m = min(70, n - a)
        assert got[32 * a:32 * (a + m)] == oracle.derive(key, source, first + a, m)
