"""A SNAP stream of as many chunks as a layer can have (2^32 boxes), which is
more than the y or z extent of a launch grid.  It takes 125 GB, so this file
comes before the ones that share the session's context."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_most_chunks():
    torch = pytest.importorskip("torch")
    from vlsi_layout_gb300 import engine
    if torch.cuda.mem_get_info()[0] < 140 << 30:
        pytest.skip("needs 140 GB of free device memory")
    chunks, per = 65_536, engine.SNAP_BOXES_PER_CHUNK
    c = torch.arange(chunks, device="cuda")
    w, h = 1 + c % 100, 101 + c // 1000 % 27
    # per chunk: a new width and height, then records that change nothing
    data = torch.zeros((chunks, per + 2), dtype=torch.uint8, device="cuda")
    data[:, 0], data[:, 1], data[:, 2] = 3 | 12, w, h
    meta = np.tile(np.array([per, per + 2, per + 2], np.int64), chunks)
    exp = torch.stack([0 * c, 0 * c, w, h], 1).to(torch.int32)
    with engine.Context(0, 64 << 20) as ctx:
        out = torch.zeros((chunks, per, 4), dtype=torch.int32, device="cuda")
        torch.cuda.synchronize()
        ctx._chk(engine.lib().gb_decompress_stream_to_boxes(ctx.h, data.data_ptr(), meta.ctypes.data, ctypes.c_int64(chunks), 0,
                                                            out.data_ptr()))
        for i in range(0, chunks, 1024):
            assert bool((out[i:i + 1024] == exp[i:i + 1024, None, :]).all()), i
    del out, data
    torch.cuda.empty_cache()
