"""A graph made on a job whose needles are replaced later: a replay runs the kernel that the new needles
call for (few needles, or regexes and many needles with their filters), like plain launches of a new job."""
import pytest

import meikey_b200 as mk
from conftest import chacha_key

pytestmark = pytest.mark.gpu

FEW = [mk.Needle.contains("q7x")]


def many():
    return ([mk.Needle.contains(t) for t in ("abcd", "efgh", "ijkl", "mnop", "qrst", "uvwx", "yzAB", "CDEF", "x7q")] +
            [mk.Needle.regex(r) for r in ("ab[0-9]", "(?:xyz|XYZ)$", "z[0-9]{2}z")])


@pytest.mark.parametrize("source", [mk.SEED_COUNTER, mk.SEED_INCREMENTAL])
@pytest.mark.parametrize("first", ["few", "many"])
def test_replays_follow_the_needles(gpu_ctx, source, first):
    key = bytearray(chacha_key(17))
    key[31] &= 0x7f
    sets = {"few": FEW, "many": many()}
    span = gpu_ctx.keys_per_iter

    def fresh(needles, base):
        with gpu_ctx.job(bytes(key), source, needles) as job:
            hits = []
            for k in range(2):
                job.launch(base + k * span, 1)
                got, total = job.hits(cap=1 << 18)
                assert total == len(got)
                hits += got
        return hits

    other = "many" if first == "few" else "few"
    with gpu_ctx.job(bytes(key), source, sets[first]) as job:
        graph = job.graph(1, 2)
        base = 2**32 + 3
        for name in (first, other, first, other):
            job.update(sets[name])
            graph.launch(base)
            got, total = job.hits(cap=1 << 18)
            want = fresh(sets[name], base)
            assert got == want and total == len(want)
            assert {k for _, k in want} >= ({0} if name == "few" else {8, 9})  # 3 characters, one regex
            base += 2 * span
        graph.close()
