"""The key filters in front of the matcher, against the oracle's exact candidate sets: the quick compare
of a few case-sensitive needles (every length and position, suffixes, the sign-dependent position 42),
and the bucket filter of many needles of 4 and more characters (the last window of a key included).
Needles are cut from keys of the range, so that each has something to find."""
import random

import pytest

import meikey_b200 as mk
from conftest import chacha_key
from meikey_b200.engine import openssh_public

pytestmark = pytest.mark.gpu

KEY, BASE, N = chacha_key(21), 2**30 + 1, 20000


@pytest.fixture(scope="module")
def tails(oracle):
    """The 44 base64 characters behind the fixed prefix of the first keys (position 0 is not searched)."""
    raw = oracle.derive(KEY, 1, BASE, 400)
    return [openssh_public(raw[32 * i:32 * i + 32]).split()[1][-44:] for i in range(400)]


def check(ctx, oracle, needles):
    with ctx.job(KEY, mk.SEED_COUNTER, needles) as job:
        job.launch(BASE, 1)
        hits, total = job.hits(cap=1 << 18)
    assert total == len(hits)
    got = sorted(h for h in hits if h[0] < BASE + N)
    want = sorted((i, k) for k, n in enumerate(needles)
                  for i in oracle.search(KEY, 1, BASE, N, n.text, len(n.text), n.fold, n.mode))
    assert got == want and {k for _, k in want} == set(range(len(needles)))


@pytest.mark.parametrize("length", [3, 4, 5, 6, 9, 20, 42])
def test_quick_contains_at_every_position(gpu_ctx, oracle, tails, length):
    rng = random.Random(length)
    for pos in {1, 2, 20, 37, 38, 39, 40, 41, 44 - length}:
        if pos + length <= 44:
            texts = [t[pos:pos + length] for t in rng.sample(tails, 2)]
            check(gpu_ctx, oracle, [mk.Needle.contains(t) for t in texts])


@pytest.mark.parametrize("length", [2, 3, 5, 6, 17, 43])
def test_quick_suffixes_beside_a_contains_needle(gpu_ctx, oracle, tails, length):
    rng = random.Random(length)
    for count in (1, 4):
        needles = [mk.Needle.suffix(t[44 - length:]) for t in rng.sample(tails, count)]
        check(gpu_ctx, oracle, needles)
        check(gpu_ctx, oracle, needles + [mk.Needle.contains(tails[0][7:11])])


@pytest.mark.parametrize("count,lo,hi", [(8, 4, 4), (9, 5, 9), (40, 4, 9), (100, 4, 5)])
def test_bucket_filter(gpu_ctx, oracle, tails, count, lo, hi):
    rng = random.Random(count)
    needles = []
    for q in range(count):
        length = rng.randint(lo, hi)
        pos = (44 - length, 41 - length if length < 9 else 30, rng.randint(1, 44 - length))[q % 3]
        text = tails[q][pos:pos + length]
        if q % 4 == 1 and pos + length == 44:
            needles.append(mk.Needle.suffix(text, case_sensitive=q % 8 == 1))
        else:
            needles.append(mk.Needle.contains(text, case_sensitive=q % 2 == 0))
    if count == 9:
        needles.append(mk.Needle.contains(tails[200][5:8]))  # scanned for every key, beside the filter
    check(gpu_ctx, oracle, needles)


REGEXES = ["ab[0-9]", "(ab|cd|ef)[+/]", "(?:xyz|XY|q[a-c])z$", "aa?b[xy]c?d$", "z[0-9]{2}z", "(?:a[ab]b|bab)[cd]", "qq+w",
           "(?i)hij", "[a-f][0-9]{2}$", "(?i)k.l.m", "zz$", "^K..x", "(ab){2}", "/[+]/", "[xyz]{5}", "(?i)[a-c]{4}$"]


@pytest.mark.parametrize("texts", [0, 1, 20])
@pytest.mark.parametrize("which", [slice(0, 16), slice(0, 5), slice(5, 10), slice(9, 11)])
def test_regexes_together_find_what_each_finds_alone(gpu_ctx, tails, which, texts):
    """A job of one regex walks its DFA for every key; several take the bucket filter."""
    def hits_of(needles):
        with gpu_ctx.job(KEY, mk.SEED_COUNTER, needles) as job:
            job.launch(BASE, 1)
            hits, total = job.hits(cap=1 << 18)
        assert total == len(hits)
        return hits

    rx = [mk.Needle.regex(r) for r in REGEXES[which]]
    text = [mk.Needle.contains(tails[q][3:8]) for q in range(texts)]
    got = hits_of(rx + text)
    for k, n in enumerate(rx):
        assert [i for i, q in got if q == k] == [i for i, _ in hits_of([n])], REGEXES[which][k]
    assert {q for _, q in got} >= set(range(len(rx), len(rx) + texts))
