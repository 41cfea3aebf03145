"""Calls at the ends of what the entry points accept, bit for bit against the
oracle: boxes that span all of int32, malformed streams of several blocks,
invalid boxes, layers used by another context or made after an error."""
import numpy as np
import pytest

from gen import random_layer

pytestmark = pytest.mark.gpu


# a tile of a warp with one and two boxes a lane, a tile of a CTA, a tile whose boxes are read from global memory
@pytest.mark.parametrize("n", [1, 5, 40, 127, 128, 300, 1023, 1500])
def test_boxes_spanning_int32(ctx, oracle, n):
    A = random_layer(n, die=40_000, wmin=20, wmax=900, seed=n)
    full = np.array([[-2**31, -2**31, 2**31 - 1, 2**31 - 1]], np.int32)
    for at in (0, n // 2, n):
        b = np.concatenate([A[:at], full, A[at:]])
        nc, lab = ctx.components(b)
        en, elab = oracle.components(b)
        assert nc == en and np.array_equal(lab, elab)
        got, exp = ctx.interactions(b), oracle.interactions(b)
        assert got[:2] == exp[:2] and np.array_equal(got[2], exp[2])
