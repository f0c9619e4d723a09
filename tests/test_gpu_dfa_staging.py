"""DFA tables in shared memory: a context of 256 threads per CTA keeps both CTAs of an SM, tables that
do not fit beside them are walked in global memory, and the candidates do not depend on it."""
import pytest

import meikey_b200 as mk
from conftest import chacha_key
from launched import kernels_of

pytestmark = pytest.mark.gpu

# tables of 9 to 57 states, 20 KB together
REGEXES = ["(ab|cd|ef)[+/]x", "(?:aa|bb)(?:cc|dd)$", "x.{2}y.{2}z", "(?:ab|ba).{2}[0-9]{2}$", "z[0-9]{3}z", "(?:xyz|XYZ)$",
           "(?:AA|BB|CC)[0-9]{3}", "[ab].{4}[cd]z[0-9]"]
MORE = ["(a.{4}b|c.{3}d)x", "x.{3}y.{2}z", "q[a-m]{3}"]  # 244, 55 and 5 states: the first alone is too large


def test_both_ctas_stay_resident():
    runs = kernels_of(f"""
        with mk.Context(device=0, table_rows=16, keys_per_thread=8, block=256) as ctx:
            with ctx.job(bytes(32), mk.SEED_COUNTER, [mk.Needle.regex(r) for r in {REGEXES!r}]) as job:
                job.launch(0, 1)
    """)
    shared, = [args["shared memory"] for name, args in runs if "k_search<" in name]
    assert 2 * (shared + 1024) <= 228 * 1024  # 228 KB of an SM, 1 KB of it reserved per CTA


@pytest.mark.parametrize("source", [mk.SEED_COUNTER, mk.SEED_INCREMENTAL])
@pytest.mark.parametrize("regexes,texts", [(REGEXES, 0), (REGEXES, 20), (MORE, 0), (MORE + REGEXES[:2], 0), (REGEXES[:1], 1)])
def test_candidates_with_some_tables_in_global_memory(gpu_ctx, source, regexes, texts):
    """Together on a context with two CTAs per SM as each alone on one of 512 threads."""
    key = bytearray(chacha_key(31))
    key[31] &= 0x7f
    base, n = 2**30 + 1, 2_000_000
    text = [mk.Needle.contains(f"{q:02d}ab") for q in range(texts)]

    def hits_of(ctx, needles):
        with ctx.job(bytes(key), source, needles) as job:
            job.launch(base, -(-n // ctx.keys_per_iter))
            hits, total = job.hits(cap=1 << 20)
        assert total == len(hits)
        return [h for h in hits if h[0] < base + n]

    rx = [mk.Needle.regex(r) for r in regexes]
    with mk.Context(device=0, table_rows=16, keys_per_thread=8, block=256, hit_capacity=1 << 20) as ctx:
        got = hits_of(ctx, rx + text)
    for k, needle in enumerate(rx + text):
        assert [i for i, q in got if q == k] == [i for i, _ in hits_of(gpu_ctx, [needle])]
    assert got
