"""Replacing a job's regexes costs about what their tables cost to copy: working out which keys can match
them (tables of up to 256 states) must not take several times as long."""
import time

import pytest

import meikey_b200 as mk
from conftest import chacha_key

pytestmark = pytest.mark.gpu


def test_update_with_filtered_regexes(gpu_ctx):
    def cost(pattern):
        needles = [mk.Needle.regex(pattern)] * 16
        with gpu_ctx.job(chacha_key(1), mk.SEED_COUNTER, needles) as job:
            def once():
                t = time.perf_counter()
                job.update(needles)
                return time.perf_counter() - t
            return needles[0].c_len(), min(once() for _ in range(50))

    states, filtered = cost("x.{5}y.{2}z")
    more_states, copied = cost("a.{7}b")
    assert states <= 256 < more_states
    assert filtered < 3 * copied
