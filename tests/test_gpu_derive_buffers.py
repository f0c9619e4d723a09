"""mk_derive into buffers of every kind of memory, short (the copy alone) and long enough for its
pages to be made present first, and the device memory that a context keeps."""
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


def test_device_memory_kept_for_later_calls():
    """The 128 MB of 4 M keys at most, in a pool that grows by 32 MB blocks, until the context goes."""
    def free_bytes():
        torch.cuda.synchronize()
        return torch.cuda.mem_get_info()[0]

    with mk.Context(device=0, table_rows=16) as ctx:
        # the kernel of 16 keys per thread has run: the driver keeps local memory for the largest so far
        ctx.derive(KEY, mk.SEED_CHACHA20, 5, 1 << 20)
    free = free_bytes()
    with mk.Context(device=0, table_rows=16) as ctx:
        ctx.derive(KEY, mk.SEED_CHACHA20, 5, 1)
        before = free_bytes()
        for n in (1 << 20, (1 << 22) + 3, 1 << 22, 1 << 23):
            got = ctx.derive(KEY, mk.SEED_CHACHA20, 5, n)
            assert before - free_bytes() <= 160 << 20
            assert got[-32:] == ctx.derive(KEY, mk.SEED_CHACHA20, 5 + n - 1, 1)
    assert free - free_bytes() <= 2 << 20
