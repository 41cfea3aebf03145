"""The work that users of the engine have it do, as timed cases.

Every case goes through a public entry point: the reference's own FFI
(boost_polygon_operation, device_event_sort), the operators on layers resident
in HBM, the host-buffer calls (op1_host, components, interactions), the
serving loop, the device sorts and the SNAP codec.  Layouts have the shapes of
the repository's configurations: random layers (lower-left uniform, sides
20..2000 dbu, die side 1e6 * sqrt(n / 1e5)), batches of such cells with
lognormal box counts, and standard-cell layers (poly stripes, met1 / met2
wires, li1 rectangles, contacts) at the density of the connectivity benchmark.

listed() gives the cases, draw(rng) another one of the same ranges,
prepare(case, seed) the inputs and handles, run(state) one pass, work(case)
the bytes and operations of a pass, exact(case, seed) its result by torch.
"""
import ctypes
import math

import numpy as np
import torch

from vlsi_layout_gb300 import engine

ARENA = 24 << 30       # work arena of the context that the resident-layer cases share
CHUNK = engine.SNAP_BOXES_PER_CHUNK
PAIRS = {"li1 x met1": ("li1", "met1"), "poly x li1": ("poly", "li1"), "met1 x met2": ("met1", "met2")}
OPS = {"xor": engine.XOR, "or": engine.OR, "and": engine.AND, "not": engine.NOT, "merge": engine.MERGE,
       "overlap": engine.OVERLAP}

# kind -> (smallest n, largest n) of drawn cases; n counts boxes (per layer for ffi, bool and serve, cells for op1)
RANGES = {"ffi": (200, 150_000), "bool": (20_000, 1_000_000), "size": (20_000, 2_000_000),
          "area": (50_000, 12_000_000), "op1": (1, 768), "components": (1_000, 4_000_000),
          "interactions": (1_000, 3_000_000), "serve": (2_000, 120_000), "morton": (1_000, 60_000_000),
          "events": (1_000, 20_000_000), "encode": (3_000, 12_000_000), "decode": (3_000, 12_000_000)}


def listed():
    return [
        # one AND between two layers of one small cell, as the Fortran layer calls it: host boxes in, host boxes out
        {"name": "ffi_and_1k", "kind": "ffi", "n": 1237, "m": 911, "op": "and", "amount": 0},
        # XOR of two mask layers of a standard-cell block, both resident, the strips read back
        {"name": "bool_xor_1m", "kind": "bool", "n": 1_000_003, "pair": "li1 x met1", "op": "xor"},
        # erosion (SIZE -s) of a random layer, the sizing step of a width check
        {"name": "size_minus_500k", "kind": "size", "n": 500_000, "amount": -7},
        # Klee's-measure area of a large layer
        {"name": "area_12m", "kind": "area", "n": 12_000_000},
        # the OP1 ring-check deck on a batch of uneven cells from pinned host memory
        {"name": "op1_1024_cells", "kind": "op1", "n": 1024},
        # PNUM connectivity of a standard-cell layout through its contacts, host boxes in, labels out
        {"name": "components_4m", "kind": "components", "n": 4_000_000},
        # overlap pairs and singletons of a block while it is loaded
        {"name": "interactions_300k", "kind": "interactions", "n": 300_001},
        # the request loop: a burst of mixed requests on resident layers of uneven size
        {"name": "serve_burst", "kind": "serve", "n": 60_000, "requests": 40},
        # Morton order of a chip-sized layer on the device
        {"name": "morton_60m", "kind": "morton", "n": 59_999_999, "die": 40_000_000, "centred": False},
        # tracker events of a sweep, sorted in place in device memory
        {"name": "events_20m", "kind": "events", "n": 20_000_000, "die": 40_000_000, "centred": False},
        # a Morton-ordered layer to SNAP chunks and back, the out-of-core path
        {"name": "snap_encode_12m", "kind": "encode", "n": 12_000_000, "method": 1},
        {"name": "snap_decode_12m", "kind": "decode", "n": 12_000_000, "method": 1},
    ]


def draw(rng):
    kind = rng.choice(sorted(RANGES))
    lo, hi = RANGES[kind]
    n = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    case = {"kind": kind, "n": n}
    if kind == "ffi":
        case.update(m=max(1, int(n * rng.uniform(0.2, 1.0))), op=rng.choice(["xor", "or", "and", "not", "merge", "size"]),
                    amount=rng.choice([-11, -3, -1, 1, 2, 9]))
    elif kind == "bool":
        case.update(pair=rng.choice(sorted(PAIRS)), op=rng.choice(sorted(OPS)))
    elif kind == "size":
        case.update(amount=rng.choice([-60, -25, -5, -1, 1, 4, 30, 75]))
        if case["amount"] < 0:
            case["n"] = min(n, 500_000)
    elif kind == "serve":
        case.update(requests=rng.randint(9, 40))
    elif kind in ("morton", "events"):
        case.update(die=rng.choice([1_000_000, 6_700_000, 40_000_000]), centred=rng.random() < 0.3)
    elif kind in ("encode", "decode"):
        case.update(method=rng.choice([0, 1, 1]))
    return case


# ------------------------------------------------------------------ layouts
def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _upto(hi, n, g, lo=0):
    """uniform int64 in [lo, hi); hi may be a tensor."""
    u = torch.rand(n, device="cuda", generator=g, dtype=torch.float64)
    return lo + (u * (hi - lo)).to(torch.int64)


def _boxes(x, y, w, h):
    return torch.stack([x, y, x + w, y + h], 1).to(torch.int32).contiguous()


def _random(n, g, die=None):
    if die is None:
        die = max(4000, int(1e6 * math.sqrt(n / 1e5)))
    w, h = _upto(2001, n, g, 20), _upto(2001, n, g, 20)
    return _boxes(_upto(die - w, n, g), _upto(die - h, n, g), w, h)


def _wire(n, die, g):
    return torch.exp(7.0 + torch.randn(n, device="cuda", generator=g, dtype=torch.float64)).round().clamp(140, die // 2).to(torch.int64)


def _stdcell(n, g):
    """dict of layers of n boxes each (contacts: n // 50)."""
    die = max(20_000, int(400_000 * math.sqrt(n / 100_000)))
    full = lambda v, k=n: torch.full((k,), v, dtype=torch.int64, device="cuda")  # noqa: E731
    L1, L2 = _wire(n, die, g), _wire(n, die, g)
    w, h = _upto(801, n, g, 170), _upto(801, n, g, 170)
    c = max(1, n // 50)
    return {"poly": _boxes(_upto(die // 340, n, g) * 340, _upto(die - 2600, n, g), full(150), _upto(2501, n, g, 500)),
            "met1": _boxes(_upto(die - L1, n, g), _upto(die // 340, n, g) * 340, L1, full(140)),
            "met2": _boxes(_upto(die // 340, n, g) * 340 + 100, _upto(die - L2, n, g), full(140), L2),
            "li1": _boxes(_upto(die - w, n, g), _upto(die - h, n, g), w, h),
            "contact": _boxes(_upto(die - 170, c, g), _upto(die - 170, c, g), full(170, c), full(170, c))}


def _block(n, g):
    """One layer of n boxes: the four standard-cell layers and 2% contacts."""
    s = _stdcell(max(1, n // 4 + 1), g)
    b = torch.cat([s[k] for k in ("contact", "poly", "met1", "met2", "li1")])
    return b[torch.randperm(b.shape[0], device="cuda", generator=g)[:n]].contiguous()


def _morton_order(b):
    """Sorted Morton keys of the box centres and the permutation that sorts them."""
    x = torch.div(b[:, 0].to(torch.int64) + b[:, 2], 2, rounding_mode="trunc") + (1 << 31)
    y = torch.div(b[:, 1].to(torch.int64) + b[:, 3], 2, rounding_mode="trunc") + (1 << 31)

    def spread(v):
        for s, m in ((16, 0x0000FFFF0000FFFF), (8, 0x00FF00FF00FF00FF), (4, 0x0F0F0F0F0F0F0F0F),
                     (2, 0x3333333333333333), (1, 0x5555555555555555)):
            v = (v | (v << s)) & m
        return v

    keys, perm = torch.sort((spread(x) | (spread(y) << 1)) ^ (-1 << 63), stable=True)  # unsigned order
    return keys ^ (-1 << 63), perm.to(torch.int32)


# ------------------------------------------------------------------ handles
_ctx = None


def _context():
    """One context per process, as a program keeps it."""
    global _ctx
    if _ctx is None:
        _ctx = engine.Context(0, ARENA)
    return _ctx


class _Layer(engine.Layer):
    """A resident layer over boxes in device memory, freed with its state."""

    def __init__(self, boxes):
        torch.cuda.synchronize()
        h = ctypes.c_void_p()
        ctx = _context()
        ctx._chk(engine.lib().gb_layer_from_device(ctx.h, boxes.data_ptr(), boxes.shape[0], None, 1, ctypes.byref(h)))
        super().__init__(ctx, h, 1)

    def __del__(self):
        self.free()


class _Server(engine.Server):
    def __del__(self):
        self.close()


def _to_pinned(layer, out):
    """The layer's strips in the pinned buffer that the program keeps for results, and their number."""
    n = ctypes.c_uint64()
    layer.ctx._chk(engine.lib().gb_layer_to_host(layer.ctx.h, layer.h, out.data_ptr(), out.shape[0], ctypes.byref(n), None))
    return out, n.value


def _pinned(n):
    return torch.zeros((n, 4), dtype=torch.int32, pin_memory=True)


# ------------------------------------------------------------------ cases
def prepare(case, seed):
    kind, n, g = case["kind"], case["n"], _gen(seed)
    s = {"case": case}
    if kind == "ffi":
        die = max(4000, int(1e6 * math.sqrt(n / 1e5)))
        s["a"], s["b"] = _random(n, g, die).cpu().numpy(), _random(case["m"], g, die).cpu().numpy()
        # the caller's result buffer, by the FFI's convention
        s["out"] = np.zeros(((10 if case["op"] == "and" else 4) * n, 4), np.int32)
    elif kind == "bool":
        layers = _stdcell(n, g)
        s["a"], s["b"] = (_Layer(layers[k]) for k in PAIRS[case["pair"]])
        s["out"] = _pinned(6 * n + 4096)
    elif kind == "size":
        s["a"] = _Layer(_random(n, g))
        s["out"] = _pinned(6 * n + 4096)
    elif kind == "area":
        s["a"] = _Layer(_random(n, g))
    elif kind == "op1":
        counts = torch.exp(math.log(8000) + 0.92 * torch.randn(n, device="cuda", generator=g, dtype=torch.float64))
        counts = counts.round().clamp(100, 100_000).to(torch.int64)
        die = (1e6 * torch.sqrt(counts / 1e5)).to(torch.int64).clamp(min=4000)
        total = int(counts.sum())
        boxes = _random(total, g, torch.repeat_interleave(die, counts))
        s["boxes"] = _pinned(total)
        s["boxes"].copy_(boxes)
        s["offsets"] = np.concatenate([[0], torch.cumsum(counts, 0).cpu().numpy()]).astype(np.int64)
    elif kind in ("components", "interactions"):
        s["boxes"] = _block(n, g).cpu().numpy()
    elif kind == "serve":
        s["server"] = _Server(0, 8 << 30, 3, 1 << 30)
        r = np.random.default_rng(seed)
        sizes = np.clip(np.round(n * r.lognormal(0.0, 0.8, 8)), 100, 250_000).astype(np.int64)
        for k in sizes:
            s["server"].add_layer(_random(int(k), g).cpu().numpy())
        q = np.zeros(case["requests"], engine.REQUEST_DTYPE)
        # every operator comes up; the burst arrives at once
        q["op"] = np.array([engine.AND, engine.NOT, engine.OR, engine.XOR, engine.REQ_SIZE, engine.REQ_GROW])[np.arange(len(q)) % 6]
        q["a"], q["b"] = r.integers(0, 8, len(q)), r.integers(0, 8, len(q))
        q["amount"] = np.where(q["op"] == engine.REQ_SIZE, r.choice([-3, -1, 2, 5], len(q)), r.integers(1, 8, len(q)))
        s["requests"] = q
    elif kind == "morton":
        s["boxes"] = _die_boxes(case, g)
        s["keys"], s["keys2"] = (torch.empty(n, dtype=torch.int64, device="cuda") for _ in range(2))
        s["vals"], s["vals2"] = (torch.empty(n, dtype=torch.int32, device="cuda") for _ in range(2))
        s["bits"] = 64 if case["centred"] else 2 * int(case["die"]).bit_length()
    elif kind == "events":
        s["events"] = _events(case, g)
    else:
        b = _block(n, g)
        b = b[_morton_order(b)[1].long()].contiguous()
        cap = ctypes.c_int64()
        engine.lib().gb_snap_max_bytes(n, ctypes.byref(cap))
        s["boxes"] = b
        s["data"] = torch.zeros(cap.value, dtype=torch.uint8, device="cuda")
        s["meta"] = np.zeros(3 * ((n + CHUNK - 1) // CHUNK), np.int64)
        _context()
        if kind == "decode":
            torch.cuda.synchronize()
            _encode(s)
            s["boxes"] = torch.zeros_like(b)
    torch.cuda.synchronize()  # the engine works on its own stream
    return s


def _die_boxes(case, g):
    """Random boxes of a die whose corner, or whose centre, is the origin."""
    b = _random(case["n"], g, case["die"])
    return b - case["die"] // 2 if case["centred"] else b


def _events(case, g):
    """n trackers of 12 bytes: X, Y, polygon number (padded with zeros)."""
    n, x0 = case["n"], case["die"] // 2 if case["centred"] else 0
    x, y = _upto(case["die"], n, g) - x0, _upto(case["die"], n, g) - x0
    return torch.stack([x, y, torch.randint(1, 5, (n,), device="cuda", generator=g)], 1).to(torch.int32).contiguous()


def _encode(s):
    ctx, total = _context(), ctypes.c_int64()
    ctx._chk(engine.lib().gb_compress_boxes_to_stream(
        ctx.h, s["boxes"].data_ptr(), s["case"]["n"], s["case"]["method"], s["data"].data_ptr(), s["data"].numel(),
        s["meta"].ctypes.data, ctypes.byref(total)))
    return s["data"], s["meta"], total.value


def run(s):
    case = s["case"]
    kind, n = case["kind"], case["n"]
    if kind == "ffi":
        op, count = engine.SIZE if case["op"] == "size" else OPS[case["op"]], ctypes.c_ulong()
        engine.lib().PerformBoostPolygonOperation(s["a"].ctypes.data, n, s["b"].ctypes.data, len(s["b"]), s["out"].ctypes.data,
                                                  ctypes.byref(count), op, case["amount"])
        return s["out"], count.value
    if kind == "bool":
        ctx = _context()
        mark = ctx.mark()
        out = _to_pinned(ctx.op(OPS[case["op"]], s["a"], s["b"]), s["out"])
        ctx.release(mark)
        return out
    if kind == "size":
        ctx = _context()
        mark = ctx.mark()
        out = _to_pinned(ctx.size(s["a"], case["amount"]), s["out"])
        ctx.release(mark)
        return out
    if kind == "area":
        ctx = _context()
        mark = ctx.mark()
        out = ctx.area(s["a"])
        ctx.release(mark)
        return out
    if kind == "op1":
        counts, area, fails, digests = _context().op1_host(s["boxes"].data_ptr(), s["boxes"].shape[0], s["offsets"], 1,
                                                           digests=True)
        return {"counts": counts, "area": area, "failures": fails, "digests": digests.view(np.int64)}
    if kind == "components":
        return _context().components(s["boxes"])
    if kind == "interactions":
        return _context().interactions(s["boxes"])
    if kind == "serve":
        r = s["server"].run(s["requests"])
        return r["status"], r["count"]
    if kind == "morton":
        ctx = _context()
        ctx._chk(engine.lib().gb_morton_keys_device(ctx.h, s["boxes"].data_ptr(), n, s["keys"].data_ptr(), s["vals"].data_ptr()))
        ctx.radix_sort_device(s["keys"].data_ptr(), s["vals"].data_ptr(), n, s["bits"], s["keys2"].data_ptr(), s["vals2"].data_ptr())
        return s["keys"], s["vals"]
    if kind == "events":
        e = s["events"].clone()  # the call sorts in place
        torch.cuda.current_stream().synchronize()  # it runs on the engine's own stream
        engine.lib().device_event_sort(e.data_ptr(), n)
        return e
    if kind == "encode":
        return _encode(s)
    ctx = _context()
    ctx._chk(engine.lib().gb_decompress_stream_to_boxes(ctx.h, s["data"].data_ptr(), s["meta"].ctypes.data,
                                                        len(s["meta"]) // 3, case["method"], s["boxes"].data_ptr()))
    return s["boxes"]


def work(case):
    """Inputs read once and outputs written once.  Strips per input box of the
    Booleans are those of the layouts above (random layers overlap a little,
    standard-cell wires a lot)."""
    kind, n = case["kind"], case["n"]
    if kind == "ffi":
        k = n + case["m"]
        return {"bytes": 16 * k + 16 * (0.5 * k if case["op"] == "and" else 2 * k), "flops": 0}
    if kind == "bool":
        k = n if case["op"] in ("merge", "overlap") else 2 * n
        return {"bytes": 16 * k + 16 * k, "flops": 0}
    if kind == "size":
        return {"bytes": 16 * n + 16 * 2 * n, "flops": 0}
    if kind == "area":
        return {"bytes": 16 * n + 8, "flops": 0}
    if kind == "op1":  # 16 B a box in; per cell six counts, six digests and the area out
        return {"bytes": n * (16 * 12_000 + 13 * 8), "flops": 0}
    if kind == "components":
        return {"bytes": 16 * n + 8 * n, "flops": 0}
    if kind == "interactions":
        return {"bytes": 16 * n + n, "flops": 0}
    if kind == "serve":
        return {"bytes": case["requests"] * 1.4 * n * (1.6 * 16 + 2 * 16), "flops": 0}
    if kind == "morton":  # the boxes in, keys and permutation out
        return {"bytes": 16 * n + 12 * n, "flops": 0}
    if kind == "events":
        return {"bytes": 12 * n + 12 * n, "flops": 0}
    return {"bytes": 16 * n + 9 * n, "flops": 0}


def exact(case, seed):
    """The sorts' and the codec's results as torch gives them; the Booleans have no such short form."""
    if case["kind"] == "morton":
        return _morton_order(_die_boxes(case, _gen(seed)))
    if case["kind"] == "events":
        e = _events(case, _gen(seed))
        key = (e[:, 0].to(torch.int64) << 32) + e[:, 1].to(torch.int64)
        return e[torch.sort(key, stable=True)[1]].contiguous()
    if case["kind"] == "decode":
        b = _block(case["n"], _gen(seed))
        return b[_morton_order(b)[1].long()].contiguous()
    return None
