"""Device memory: calls run in what they need, and what one context's pool keeps
is there for others."""
import numpy as np
import pytest

from gen import random_layer

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def _leave(free):
    """Takes device memory until `free` bytes are left."""
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    return torch.empty(torch.cuda.mem_get_info()[0] - free, dtype=torch.uint8, device="cuda")


def test_morton_sort_memory(oracle):
    """44 bytes a box: boxes, keys and values, then the sort's buffers or the sorted boxes (64 in one allocation)."""
    from vlsi_layout_gb300 import engine
    n = 20_000_000
    A = random_layer(n, die=3_000_000, seed=1)
    with engine.Context(0, 64 << 20) as ctx:
        ctx.morton_sort(A[:1_000_000])
        ballast = _leave(n * 54)
        try:
            b, keys, perm = ctx.morton_sort(A)
        finally:
            del ballast
            torch.cuda.empty_cache()
    k = oracle.morton_keys_np(A)
    assert np.array_equal(perm, np.argsort(k, kind="stable"))
    assert np.array_equal(keys, k[perm]) and np.array_equal(b, A[perm])
