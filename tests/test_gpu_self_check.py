"""The self-check at context creation covers every derive kernel: each number of keys per thread, for
hashed seeds and the incremental source, as calls of different lengths use them."""
import re

import pytest

from launched import kernels_of

pytestmark = pytest.mark.gpu


def test_every_derive_kernel_is_checked():
    names = [n for n, _ in kernels_of("mk.Context(device=0, table_rows=16, keys_per_thread=4, self_check=True).close()")]
    got = {m.groups() for n in names if (m := re.search(r"k_derive<(\d+), (true|false)>", n))}
    assert got == {(str(k), incr) for k in (1, 2, 4, 8, 16) for incr in ("true", "false")}
