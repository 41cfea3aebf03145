"""Calls at the ends of what the entry points accept, bit for bit against the
oracle: boxes that span all of int32, malformed streams of several blocks,
invalid boxes, layers used by another context or made after an error."""
import time

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


def _indexed_stream(at, index, height, n=65536):
    """A valid chunk and one of n records: a new width and height, then records that change nothing, but record `at`,
    which sets the width (height) to the dictionary's entry `index`."""
    raw = bytearray([3 | 12, 10, 20]) + bytes(n - 1)
    rec = bytes([4 if height else 1]) + (index & 0xFFFF).to_bytes(2, "little")
    bad = bytes(raw[:at + 2]) + rec + bytes(raw[at + 3:])
    return [(65536, 65538, 65538, bytes(raw[:65538])), (n, len(bad), len(bad), bad)]


# records of the first, a middle and the last block of 1024; entries that do not exist, the only one that does
@pytest.mark.parametrize("at", [1, 1023, 40_000, 65_535])
@pytest.mark.parametrize("height", [False, True])
def test_stream_dictionary_index(ctx, oracle, at, height):
    from vlsi_layout_gb300 import engine
    ok = _indexed_stream(at, 1, height)
    b = ctx.decompress_stream_to_boxes(ok, 0)
    assert np.array_equal(b, np.tile(np.array([[0, 0, 10, 20]], np.int32), (131_072, 1)))
    for index in (0, 2, 30_000, 32_767, -1, -32_768):
        bad = _indexed_stream(at, index, height)
        with pytest.raises(ValueError):
            oracle.codec_decode_chunk(bad[1][3], 65536)
        with pytest.raises(engine.GBError) as e:
            ctx.decompress_stream_to_boxes(bad, 0)
        assert e.value.code == engine.GB_ERR_CORRUPT, index
    assert np.array_equal(ctx.decompress_stream_to_boxes(ok, 0), b)


@pytest.mark.parametrize("nbad", [1, 40, 3000])
def test_invalid_boxes_on_upload(oracle, nbad):
    """Invalid boxes that many blocks meet at once are an error, of the layer's every use, and the context goes on."""
    from vlsi_layout_gb300 import engine
    A = random_layer(300_000, die=1_500_000, seed=nbad)
    bad = A.copy()
    at = np.random.default_rng(nbad).choice(len(A), nbad, replace=False)
    bad[at, 2] = bad[at, 0]
    off = np.linspace(0, len(A), 701).astype(np.int64)
    exp = oracle.union_area(A)
    with engine.Context(0, 2 << 30) as ctx:
        good = ctx.layer(A)
        for cells in (None, off):
            for _ in range(10):
                m = ctx.mark()
                L = ctx.layer(bad, cells)
                with pytest.raises(engine.GBError) as e:
                    ctx.sync()
                assert e.value.code == engine.GB_ERR_INVALID_BOX
                with pytest.raises(engine.GBError) as e:
                    ctx.area(L)
                assert e.value.code == engine.GB_ERR_INVALID_BOX
                L.free()
                ctx.release(m)
            assert int(ctx.area(good)[0]) == exp


def _best(fn, k=4):
    """Shortest of k times, after a first run."""
    fn()
    ts = []
    for _ in range(k):
        t = time.perf_counter()
        fn()
        ts.append(time.perf_counter() - t)
    return min(ts)


def test_layer_made_after_an_error(ctx, oracle):
    """A layer uploaded before an error is cleared is as good as another, and as fast."""
    from vlsi_layout_gb300 import engine
    A = random_layer(400_000, die=1_700_000, seed=8)
    m = ctx.mark()
    before = ctx.layer(A)
    broken = ctx.layer(np.array([[5, 5, 1, 1]], np.int32))
    after = ctx.layer(A)
    with pytest.raises(engine.GBError):
        ctx.sync()
    exp = oracle.union_area(A)

    def area(L):
        k = ctx.mark()
        assert int(ctx.area(L)[0]) == exp
        ctx.release(k)

    assert _best(lambda: area(after)) < 20 * _best(lambda: area(before))
    for L in (before, broken, after):
        L.free()
    ctx.release(m)


def test_layer_used_by_another_context(ctx, oracle):
    """A layer is complete when the call that makes it returns: another context's stream may use it at once."""
    from vlsi_layout_gb300 import engine
    A = random_layer(1_500_000, die=3_000_000, seed=6)
    A = A[np.argsort(A[:, 0], kind="stable")]  # the last boxes widen the bounds
    exp = oracle.union_area(A)
    with engine.Context(0, 4 << 30) as other:
        for _ in range(4):
            m, k = ctx.mark(), other.mark()
            L = ctx.layer(A)
            assert int(other.area(L)[0]) == exp
            L.free()
            ctx.release(m)
            other.release(k)


def _rows(n, pitch, row, side=100):
    """Squares in rows, in the order they are drawn: records of one length."""
    i = np.arange(n, dtype=np.int64)
    x, y = i % row * pitch, i // row * pitch
    return np.stack([x, y, x + side, y + side], 1).astype(np.int32)


# pitches whose records also parse out of step, over the whole chunk or from row to row; a chain that ends in the middle
# of a chunk, at its last record and behind it
@pytest.mark.parametrize("pitch,row", [(240, 256), (240, 70_001), (500, 90), (1008, 1000), (16, 4096), (400, 256)])
@pytest.mark.parametrize("method", [0, 1])
def test_stream_out_of_step(ctx, oracle, pitch, row, method):
    from vlsi_layout_gb300 import engine
    b = _rows(70_001, pitch, row)
    chunks = oracle.stream_encode(b, method)
    assert np.array_equal(ctx.decompress_stream_to_boxes(chunks, method), b)
    if method == 0:
        raw, n = chunks[0][3], 65536
        for cut in (len(raw) - 1, len(raw) // 2, 200):  # the stream, or its last records, end early
            for tail in (b"", b"\x20" + b"\xff" * 11, b"\x60" * 50):
                data = raw[:cut] + tail
                try:
                    exp = oracle.codec_decode_chunk(data, n)
                except ValueError:
                    with pytest.raises(engine.GBError) as e:
                        ctx.decompress_stream_to_boxes([(n, len(data), len(data), data)], 0)
                    assert e.value.code == engine.GB_ERR_CORRUPT, (cut, tail)
                else:
                    assert np.array_equal(ctx.decompress_stream_to_boxes([(n, len(data), len(data), data)], 0), exp)
        data = raw + b"\x20" + b"\xff" * 11  # nothing behind the last record is read
        assert np.array_equal(ctx.decompress_stream_to_boxes([(n, len(data), len(data), data)], 0), b[:n])


def test_stream_out_of_step_time(ctx):
    """Rows whose records also parse out of step decode in the time of others (they took some 3000 times that)."""
    def seconds(pitch):
        b = _rows(1_000_000, pitch, 1000)
        chunks = ctx.compress_boxes_to_stream(b, 0)
        return _best(lambda: ctx.decompress_stream_to_boxes(chunks, 0, as_tensor=True))

    assert seconds(240) < 5 * seconds(340)


def _full_arena():
    """A context, a layer, and how many MERGEs of it its arena holds (3 at least)."""
    from vlsi_layout_gb300 import engine
    ctx = engine.Context(0, 96 << 20)
    L = ctx.layer(random_layer(150_000, die=1_000_000, seed=2))
    m, k = ctx.mark(), 0
    try:
        while True:
            ctx.op(4, L)
            ctx.sync()
            k += 1
    except engine.GBError as e:
        assert e.code == engine.GB_ERR_CAPACITY and k >= 3
    ctx.release(m)
    return ctx, L, k


def test_captured_release():
    """A release in a graph goes back to its own mark, not to a later one of the same depth."""
    from vlsi_layout_gb300 import engine
    ctx, L, k = _full_arena()
    m = ctx.mark()
    ctx.op(4, L)
    ctx.graph_begin()
    ctx.release(m)
    g = ctx.graph_end()
    for _ in range(2):
        m = ctx.mark()  # behind the first result, where k more do not fit
        ctx.graph_launch(g)
        for _ in range(k):
            ctx.op(4, L)
        ctx.sync()
        ctx.release(m)
    engine.lib().gb_graph_destroy(g)
    L.free()
    ctx.close()


def test_many_marks():
    """More marks than are kept on the device, released one by one and in one go."""
    ctx, L, k = _full_arena()
    marks = [ctx.mark() for _ in range(200)]
    ctx.op(4, L)
    for m in marks[:100:-1]:
        ctx.release(m)
    ctx.op(4, L)
    ctx.release(marks[0])
    for _ in range(k):
        ctx.op(4, L)
    ctx.sync()
    L.free()
    ctx.close()


# empty tiles between, before and behind the others: fewer and many more tiles than the kernel has CTAs
@pytest.mark.parametrize("tiles,n", [(3, 2), (40, 7), (60, 900), (300, 2), (300, 5000), (1000, 400)])
def test_sparse_layers(ctx, oracle, tiles, n):
    rng = np.random.default_rng(tiles + n)
    side = tiles * 65536

    def layer(k):
        p = rng.integers(-side // 2, side // 2 - 70_000, (k, 2))
        b = np.concatenate([p, p + rng.integers(20, 60_000, (k, 2))], 1)
        b[:2] = [[-side // 2, -side // 2, -side // 2 + 9, -side // 2 + 5], [side // 2 - 9, side // 2 - 5, side // 2, side // 2]]
        return b.astype(np.int32)

    A, B = layer(n), layer(n)
    for op in (0, 2, 3, 4):
        m = ctx.mark()
        got = ctx.op(op, ctx.layer(A), ctx.layer(B) if op != 4 else None).to_numpy()
        ctx.release(m)
        exp = oracle.boolean(A, B, op) if op != 4 else oracle.merge(A)
        assert np.array_equal(got[np.lexsort((got[:, 3], got[:, 2], got[:, 1], got[:, 0]))], exp), op
    m = ctx.mark()
    assert int(ctx.area(ctx.layer(A))[0]) == oracle.union_area(A)
    both = ctx.area(ctx.layer(np.concatenate([A, B]), [0, len(A), len(A), 2 * len(A)]))
    assert [int(a) for a in both] == [oracle.union_area(A), 0, oracle.union_area(B)]
    ctx.release(m)


# y ranks of a tile around what the buffers of one warp (188 words, wide form 420), two, four and eight warps hold (844,
# 1724, 2052 words); few columns a sub-band and many
@pytest.mark.parametrize("n", [3008, 3009, 6720, 6721, 13504, 13505, 27584, 27585, 32000])
def test_y_rank_limits(ctx, oracle, n):
    rng = np.random.default_rng(n)
    y = rng.permutation(32_000)[:n] * 2
    for width in (40, 900):
        x = rng.integers(0, 65_536 - width, n)
        A = np.stack([x, y, x + rng.integers(1, width, n), y + 1], 1).astype(np.int32)
        m = ctx.mark()
        L = ctx.layer(A)
        got = ctx.op(4, L).to_numpy()
        assert np.array_equal(got[np.lexsort((got[:, 3], got[:, 2], got[:, 1], got[:, 0]))], oracle.merge(A))
        assert int(ctx.area(L)[0]) == oracle.union_area(A)
        ctx.release(m)
