"""mk_derive into buffers of every kind of memory, short (the copy alone) and long enough for its
pages to be made present first."""
import ctypes

import pytest
import torch

import meikey_b200 as mk
from conftest import chacha_key

pytestmark = pytest.mark.gpu

KEY = chacha_key(13)


def derive_into(ctx, n, address):
    return ctx._lib.mk_derive(ctx._ptr, KEY, mk.SEED_CHACHA20, 5, n, ctypes.c_void_p(address))


@pytest.mark.parametrize("n", [100, 262144, 300001])
@pytest.mark.parametrize("kind", ["pageable", "pinned", "device"])
def test_kinds_of_memory(gpu_ctx, n, kind):
    out = torch.zeros(32 * n, dtype=torch.uint8, device="cuda" if kind == "device" else "cpu",
                      pin_memory=kind == "pinned")
    torch.cuda.synchronize()
    assert derive_into(gpu_ctx, n, out.data_ptr()) == 0
    torch.cuda.synchronize()
    assert out.cpu().numpy().tobytes() == gpu_ctx.derive(KEY, mk.SEED_CHACHA20, 5, n)
