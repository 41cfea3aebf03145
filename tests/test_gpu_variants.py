"""The branches of the binning and scanline kernels at the sizes where they
change over: shared or global tile counters, boxes over many tiles, sub-bands
of a tile with more columns or y ranks than a warp's buffer holds at each
level, value tables on chip or in the scratch.  Everything bit for bit against the oracle."""
import numpy as np
import pytest

from gen import random_layer

pytestmark = pytest.mark.gpu


def canon(b):
    b = np.asarray(b, np.int32).reshape(-1, 4)
    return b[np.lexsort((b[:, 3], b[:, 2], b[:, 1], b[:, 0]))] if len(b) else b


def run(ctx, fn):
    m = ctx.mark()
    try:
        return canon(fn().to_numpy())
    finally:
        ctx.release(m)


# n around the shared-counter minimum (32768); dies of few tiles, of more tiles than shared counters (8192);
# boxes over 33 tiles and more, fewer and more of them than a block holds (64)
@pytest.mark.parametrize("n,die,nwide", [(32767, 400_000, 0), (32768, 400_000, 1), (33000, 6_100_000, 3),
                                         (40001, 900_000, 65), (700, 3_000_000, 130), (1, 5_000_000, 1)])
def test_binning(ctx, oracle, n, die, nwide):
    A = random_layer(n, die=die, seed=n)
    rng = np.random.default_rng(n)
    y = rng.integers(-die // 2, die // 2, nwide)
    wide = np.stack([np.full(nwide, -die // 2) + np.arange(nwide), y, np.full(nwide, die // 2), y + 9], 1).astype(np.int32)
    A = np.concatenate([A, wide])[rng.permutation(n + nwide)]
    assert np.array_equal(run(ctx, lambda: ctx.op(4, ctx.layer(A))), oracle.merge(A))
    m = ctx.mark()
    assert int(ctx.area(ctx.layer(A))[0]) == oracle.union_area(A)
    ctx.release(m)
    nc, lab = ctx.components(A)
    en, elab = oracle.components(A)
    assert nc == en and np.array_equal(lab, elab)


def test_binning_cells(ctx, oracle):
    """Cells of 0 .. 700 boxes: chunks that start and end inside cells, runs of empty cells."""
    rng = np.random.default_rng(4)
    counts = rng.choice([0, 1, 2, 31, 32, 33, 700], 400)
    off = np.concatenate([[0], np.cumsum(counts)])
    A = random_layer(int(off[-1]), die=150_000, seed=9, x0=-70_000, y0=-70_000)
    m = ctx.mark()
    area = ctx.area(ctx.layer(A, off))
    ctx.release(m)
    assert [int(a) for a in area] == [oracle.union_area(A[off[k]:off[k + 1]]) if counts[k] else 0 for k in range(len(counts))]


# columns of a sub-band around the buffers of levels 0..3 (128, 288, 640, 1024)
@pytest.mark.parametrize("wires", [64, 65, 144, 145, 320, 321, 512, 513, 700])
def test_wide_subbands(ctx, oracle, wires):
    i = np.arange(wires)
    A = np.stack([50 + 3 * (i % 7), 7 * i, 60_000 - (i % 11), 7 * i + 3], 1).astype(np.int32)
    B = random_layer(400, die=9000, wmin=3, wmax=400, seed=wires)
    for op in (0, 2, 3, 4):
        got = run(ctx, lambda: ctx.op(op, ctx.layer(A), ctx.layer(B) if op != 4 else None))
        assert np.array_equal(got, oracle.boolean(A, B, op) if op != 4 else oracle.merge(A)), op
    C = np.concatenate([A, B, A[::3]])
    assert np.array_equal(run(ctx, lambda: ctx.op(7, ctx.layer(C))), oracle.boolean(C, C[:0], 7))


# y ranks of a tile around the bitmaps of levels 0..3 (188, 320, 640, 2052 words)
@pytest.mark.parametrize("n", [2900, 3300, 5500, 7000, 11000, 16000])
def test_many_y_ranks(ctx, oracle, n):
    rng = np.random.default_rng(n)
    y = rng.permutation(32_000)[:n] * 2
    x = rng.integers(0, 65_000, n)
    A = np.stack([x, y, x + rng.integers(1, 500, n), y + 1], 1).astype(np.int32)
    B = random_layer(500, die=65_000, wmin=20, wmax=3000, seed=n)
    for op in (0, 3):
        assert np.array_equal(run(ctx, lambda: ctx.op(op, ctx.layer(A), ctx.layer(B))), oracle.boolean(A, B, op)), op


# distinct x and y values of a tile around what its 16-bit tables hold on chip (4474 of each), and with more
# sub-bands than on-chip counters (256); the first value is the tile's start, the last its end
@pytest.mark.parametrize("n", [4473, 4474, 4475, 4476, 16130, 16131, 18000])
def test_value_tables(ctx, oracle, n):
    rng = np.random.default_rng(n)
    v = [np.sort(np.concatenate([[0, 65536], rng.permutation(np.arange(1, 65536))[:n - 2]])) for _ in range(2)]
    i = np.unique(np.append(np.arange(0, n - 1, 2), n - 2))
    j = rng.permutation(i)
    A = np.stack([v[0][i], v[1][j], v[0][i + 1], v[1][j + 1]], 1).astype(np.int32)
    p, q = np.sort(rng.choice(n, (30, 2)), 1), np.sort(rng.choice(n, (30, 2)), 1)
    k = (p[:, 0] < p[:, 1]) & (q[:, 0] < q[:, 1])
    B = np.stack([v[0][p[k, 0]], v[1][q[k, 0]], v[0][p[k, 1]], v[1][q[k, 1]]], 1).astype(np.int32)
    for op in (0, 3):
        assert np.array_equal(run(ctx, lambda: ctx.op(op, ctx.layer(A), ctx.layer(B))), oracle.boolean(A, B, op)), op
    m = ctx.mark()
    assert int(ctx.area(ctx.layer(A))[0]) == oracle.union_area(A)
    ctx.release(m)


def _snap_cases():
    rng = np.random.default_rng(5)
    out = {}
    for n in (1, 1023, 1024, 1025, 2049, 65535, 65536, 65537, 70001):
        out["random %d" % n] = random_layer(n, die=300_000, seed=n, x0=-150_000, y0=-150_000)
    i = np.arange(70_000)
    # one-byte records; records whose bytes also parse out of step (20 a0 20 ...)
    out["equal boxes"] = np.tile(np.array([[5, 6, 15, 16]], np.int32), (70_000, 1))
    out["out of step"] = np.stack([2064 * i, 0 * i, 2064 * i + 10, 0 * i + 10], 1).astype(np.int32)
    x = rng.integers(-2**31, 2**31 - 1, (5000, 4), dtype=np.int64)  # longest records
    out["long records"] = np.stack([np.minimum(x[:, 0], x[:, 2]), np.minimum(x[:, 1], x[:, 3]),
                                    np.maximum(x[:, 0], x[:, 2]) + 1, np.maximum(x[:, 1], x[:, 3]) + 1], 1).astype(np.int32)
    sq = random_layer(70_000, die=300_000, seed=3)  # squares with a rare other box: far back to the last height
    sq[:, 2:] = sq[:, :2] + (sq[:, 2:3] - sq[:, 0:1])
    sq[[0, 30_000, 64_000], 3] += 3
    out["squares"] = sq
    return out


@pytest.mark.parametrize("case", list(_snap_cases()))
@pytest.mark.parametrize("method", [0, 1])
def test_snap_sizes(ctx, oracle, case, method):
    b = _snap_cases()[case]
    chunks = ctx.compress_boxes_to_stream(b, method)
    assert [c[3] for c in chunks] == [c[3] for c in oracle.stream_encode(b, method)]
    assert np.array_equal(ctx.decompress_stream_to_boxes(chunks, method), b)


# one CTA up to 8192 keys, tiles of 4096, 6144 and 8192 above; digits of 1 to 9 bits
@pytest.mark.parametrize("n", [2, 31, 512, 513, 8191, 8192, 8193, 65535, 65536, (1 << 21) - 1, 1 << 21])
@pytest.mark.parametrize("bits", [1, 9, 10, 19, 52, 64])
def test_radix_sizes(ctx, n, bits):
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(n + bits)
    k = rng.integers(0, 1 << 63, n, dtype=np.uint64) << np.uint64(1) | rng.integers(0, 2, n, dtype=np.uint64)
    v = rng.permutation(n).astype(np.uint32)
    order = np.argsort(k & np.uint64((1 << bits) - 1), kind="stable")
    dk, dv = torch.from_numpy(k.view(np.int64)).cuda(), torch.from_numpy(v.view(np.int32)).cuda()
    tk, tv = torch.empty_like(dk), torch.empty_like(dv)
    torch.cuda.synchronize()
    ctx.radix_sort_device(dk.data_ptr(), dv.data_ptr(), n, bits, tk.data_ptr(), tv.data_ptr())
    ctx.sync()
    assert np.array_equal(dk.cpu().numpy().view(np.uint64), k[order])
    assert np.array_equal(dv.cpu().numpy().view(np.uint32), v[order])


@pytest.mark.parametrize("n", [2, 8192, 100_003])
@pytest.mark.parametrize("lo,hi", [((0, 0), (40_000_000, 40_000_000)), ((-2**31, -2**31), (2**31 - 1, 2**31 - 1)),
                                   ((-5, 7), (-4, 8)), ((-70_000, 3), (80_000, 4)), ((9, -300), (10, 300))])
def test_event_ranges(n, lo, hi):
    from vlsi_layout_gb300 import engine
    rng = np.random.default_rng(n)
    t = np.zeros(n, engine.TRACKER_DTYPE)
    t["X"], t["Y"] = rng.integers(lo[0], hi[0], n), rng.integers(lo[1], hi[1], n)
    t["polygonNumber"] = rng.integers(-128, 128, n)
    t["pad"] = rng.integers(-128, 128, (n, 3))
    exp = t[np.lexsort((t["Y"], t["X"]))]
    assert engine.event_sort(t).tobytes() == exp.tobytes()


# tiles shared by 8, 4, 2 and 1 CTAs; wires that run through every share of a tile, and a tile with one sub-band
@pytest.mark.parametrize("side", [1, 2, 6, 7, 9, 10, 13, 14, 15, 20])
def test_shared_tiles(ctx, oracle, side):
    die, rng = side * 65536, np.random.default_rng(side)
    n = 120 * side * side
    A = random_layer(n, die=die, wmin=20, wmax=2500, seed=side)
    y = np.sort(rng.integers(0, die - 40, 60 * side))
    wires = np.stack([rng.integers(0, 3000, len(y)), y, die - rng.integers(0, 3000, len(y)), y + rng.integers(1, 30, len(y))],
                     1).astype(np.int32)
    A = np.concatenate([A, wires, [[5, 5, 9, 9]]]).astype(np.int32)
    B = random_layer(n // 2 + 1, die=die, seed=side + 100)
    for op in (0, 1, 2, 3, 4):
        got = run(ctx, lambda: ctx.op(op, ctx.layer(A), ctx.layer(B) if op != 4 else None))
        assert np.array_equal(got, oracle.boolean(A, B, op) if op != 4 else oracle.merge(A)), op
    assert np.array_equal(run(ctx, lambda: ctx.op(7, ctx.layer(A))), oracle.boolean(A, A[:0], 7))
    assert np.array_equal(run(ctx, lambda: ctx.size(ctx.layer(A), -6)), oracle.size(A, -6))
    m = ctx.mark()
    assert int(ctx.area(ctx.layer(A))[0]) == oracle.union_area(A)
    ctx.release(m)


def test_shared_tile_capacity(oracle):
    """A scratch that one CTA's share outgrows: the op is retried or spills, and stays exact."""
    from vlsi_layout_gb300 import engine
    A = random_layer(6000, die=60_000, wmin=20, wmax=9000, seed=1)
    B = random_layer(6000, die=60_000, wmin=20, wmax=9000, seed=2)
    with engine.Context(0, 1 << 30) as ctx:
        ctx._chk(engine.lib().gb_set_tile_scratch(ctx.h, 64 << 10))
        got = run(ctx, lambda: ctx.op(0, ctx.layer(A), ctx.layer(B)))
    assert np.array_equal(got, oracle.boolean(A, B, 0))
