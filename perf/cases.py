"""The work that users of the library have it do, as cases that can be timed and compared.

A user hashes images (H: one, a few, a batch; luma or colour; the default kernel or the
pdqhash-faithful one), matches hashes against a device-resident database (M: one image's 8
hashes, a few images', a whole batch's) and screens images end to end (S: one call from host
memory, or a stream of requests through the server). Images are the seeded blob images of
the benchmark (a base, 8 Gaussian blobs, N(0, 2) noise), with some noise and constant images
among them; databases hold rows of exactly 128 set bits, a few of them near-duplicates of
the queries, or clusters of near-duplicates (the benchmark's heavy-hit database).
"""
import ctypes
import math

import numpy as np
import torch

from __graft_entry__ import load_package

yp = load_package()

IMAGE_BYTES = {"f32": 1 << 20, "u8": 1 << 18, "rgb8": 3 << 18, "rgba8": 1 << 20}
KINDS = {"f32": yp._lib.INPUT_F32, "u8": yp._lib.INPUT_U8, "rgb8": yp._lib.INPUT_RGB8,
         "rgba8": yp._lib.INPUT_RGBA8}
JAROSZ = 0x200  # YPDQ_COMPRESS_JAROSZ
MEMBERS = 1000  # rows per cluster of the clustered database

_context = None


def context():
    """The program's one context (a user creates it once)."""
    global _context
    if _context is None:
        torch.cuda.init()
        _context = yp.Context(0)
    return _context


def listed():
    return [
        # one f32 luma image: what a caller who hashes as images come in waits for
        {"name": "hash_f32_1", "op": "hash", "input": "f32", "n": 1, "filter": "tent"},
        # a small ragged batch of byte images: a serving step, a video second
        {"name": "hash_u8_37", "op": "hash", "input": "u8", "n": 37, "filter": "tent"},
        # the benchmark's step
        {"name": "hash_f32_1024", "op": "hash", "input": "f32", "n": 1024, "filter": "tent"},
        # bulk hashing of decoded luma images (a backfill)
        {"name": "hash_u8_4096", "op": "hash", "input": "u8", "n": 4096, "filter": "tent"},
        # bulk hashing of colour images, a ragged batch
        {"name": "hash_rgb8_801", "op": "hash", "input": "rgb8", "n": 801, "filter": "tent"},
        # hashing with the pdqhash-faithful filter (hashes that have to agree with pdqhash's)
        {"name": "hash_jarosz_u8_1500", "op": "hash", "input": "u8", "n": 1500, "filter": "jarosz"},
        # one image's 8 hashes against a small database, hits to the host: an interactive lookup
        {"name": "match_8q_100k", "op": "match", "queries": 8, "rows": 100_000, "threshold": 31},
        # eight images' hashes against the 10M-row database
        {"name": "match_64q_10M", "op": "match", "queries": 64, "rows": 10_000_000, "threshold": 31},
        # the benchmark's step: 1,024 images' hashes against 10M rows, hits left on the device
        {"name": "scan_8192q_10M", "op": "scan", "queries": 8192, "rows": 10_000_000,
         "threshold": 31, "clustered": False},
        # 128 images' hashes against 100M clustered rows: ~1M hits, sorted on the device
        {"name": "scan_1024q_100M", "op": "scan", "queries": 1024, "rows": 100_000_000,
         "threshold": 31, "clustered": True},
        # one image from host memory to sorted hits: the end-to-end example's loop body
        {"name": "screen_f32_1", "op": "screen", "input": "f32", "n": 1, "rows": 10_000_000,
         "threshold": 31},
        # a closed loop of requests of 1-64 byte images through the server
        {"name": "serve_u8_96", "op": "serve", "input": "u8", "requests": 96, "rows": 10_000_000,
         "threshold": 31},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["hash", "hash", "hash", "match", "scan", "screen", "serve"])
    if op == "hash":
        flt = rng.choice(["tent", "tent", "tent", "jarosz"])
        kind = rng.choice(["f32", "u8", "rgb8", "rgba8"])
        hi = 1500 if flt == "jarosz" else 4096 if kind == "u8" else 1024
        return {"op": op, "input": kind, "n": _log_int(rng, 1, hi), "filter": flt}
    if op == "match":
        return {"op": op, "queries": 8 * _log_int(rng, 1, 64), "rows": _log_int(rng, 50_000, 20_000_000),
                "threshold": rng.choice([16, 31, 31, 36])}
    if op == "scan":
        if rng.random() < 0.5:
            return {"op": op, "queries": 8 * _log_int(rng, 1, 128), "rows": _log_int(rng, 1_000_000, 100_000_000),
                    "threshold": rng.choice([16, 31]), "clustered": True}
        return {"op": op, "queries": 8 * _log_int(rng, 1, 1024), "rows": _log_int(rng, 100_000, 10_000_000),
                "threshold": rng.choice([16, 31, 31, 36]), "clustered": False}
    if op == "screen":
        return {"op": op, "input": rng.choice(["f32", "u8", "rgb8"]), "n": _log_int(rng, 1, 200),
                "rows": _log_int(rng, 100_000, 10_000_000), "threshold": 31}
    return {"op": op, "input": "u8", "requests": _log_int(rng, 8, 96),
            "rows": _log_int(rng, 1_000_000, 10_000_000), "threshold": 31}


# ------------------------------------------------------------------------------- inputs

def _luma(n, gen):
    """n luma images [n, 512, 512] f32 on the GPU, clamped to [0, 255]: blob images, every
    16th noise and every 32nd (after the 24th) one constant value."""
    def u(shape, lo, hi):
        return torch.rand(shape, generator=gen, device="cuda") * (hi - lo) + lo

    base, cx, cy = u((n, 1, 1), 60, 190), u((n, 8, 1), 0, 512), u((n, 8, 1), 0, 512)
    two_s2, amp = 2 * u((n, 8, 1), 20, 120) ** 2, u((n, 8, 1), -80, 80)
    x = torch.arange(512, device="cuda", dtype=torch.float32)
    gx, gy = torch.exp(-((x - cx) ** 2) / two_s2), torch.exp(-((x - cy) ** 2) / two_s2)
    img = torch.bmm((amp * gy).transpose(1, 2), gx).add_(base)
    img.add_(torch.randn(img.shape, generator=gen, device="cuda"), alpha=2.0)
    img[8::16] = u((len(range(8, n, 16)), 512, 512), 0, 255)
    img[24::32] = torch.floor(u((len(range(24, n, 32)), 1, 1), 0, 256))
    return img.clamp_(0, 255)


def _images(kind, n, seed):
    """n images of `kind` on the GPU, made 128 at a time."""
    gen = torch.Generator(device="cuda").manual_seed(seed)
    shape = {"f32": (), "u8": (), "rgb8": (3,), "rgba8": (4,)}[kind]
    out = torch.empty((n, 512, 512) + shape, device="cuda",
                      dtype=torch.float32 if kind == "f32" else torch.uint8)
    for s in range(0, n, 128):
        m = min(128, n - s)
        if not shape:
            img = _luma(m, gen)
            out[s:s + m] = img if kind == "f32" else img.round_()
            continue
        for c in range(3):
            out[s:s + m, :, :, c] = _luma(m, gen).round_()
        if shape == (4,):
            out[s:s + m, :, :, 3] = torch.randint(0, 256, (m, 512, 512), generator=gen, device="cuda")
    return out


def _pinned(images):
    """The images in page-locked host memory, where a decoder writes them."""
    host = yp.PinnedArray(context(), tuple(images.shape),
                          np.float32 if images.dtype == torch.float32 else np.uint8)
    torch.from_numpy(host.array).copy_(images)
    return host


class _Rows:
    """Database rows [n, 32] u8 in a torch tensor, as yp.Database takes device memory."""

    def __init__(self, tensor):
        self.tensor = tensor
        self.ptr = ctypes.c_void_p(tensor.data_ptr())


def _synth_rows(n, seed):
    """n rows of exactly 128 set bits."""
    ctx = context()
    rows = torch.empty((n, 32), dtype=torch.uint8, device="cuda")
    yp._lib.check(ctx.lib.ypdq_synth_rows(ctx.handle, _ptr(rows), n, 0, seed, None))
    return rows


def _plant(rows, queries, count, seed):
    """`count` rows become copies of queries at distances 0..31 from them."""
    gen = torch.Generator(device="cuda").manual_seed(seed)
    count = min(count, rows.shape[0])
    pos = torch.randperm(rows.shape[0], generator=gen, device="cuda")[:count]
    qid = torch.randint(0, queries.shape[0], (count,), generator=gen, device="cuda")
    dist = torch.randint(0, 32, (count, 1), generator=gen, device="cuda")
    order = torch.rand((count, 256), generator=gen, device="cuda").argsort(1).argsort(1)
    bits = (order < dist).view(count, 32, 8).to(torch.uint8)
    weight = torch.tensor([1 << b for b in range(8)], dtype=torch.uint8, device="cuda")
    rows[pos] = queries[qid] ^ (bits * weight).sum(2).to(torch.uint8)


def _clustered(n_rows, n_queries, seed):
    """(rows, queries): clusters of MEMBERS rows each within ~20 bits of their centre, and
    the queries, which are centres."""
    ctx = context()
    rows = torch.empty((n_rows, 32), dtype=torch.uint8, device="cuda")
    yp._lib.check(ctx.lib.ypdq_synth_clustered_rows(ctx.handle, _ptr(rows), n_rows, 0, MEMBERS, 40,
                                                    seed, None))
    centres = _synth_rows(max(n_rows // MEMBERS, n_queries), seed)
    gen = torch.Generator(device="cuda").manual_seed(seed)
    pick = torch.randperm(centres.shape[0], generator=gen, device="cuda")[:n_queries]
    return rows, centres[pick].contiguous()


def _ptr(tensor):
    return ctypes.c_void_p(tensor.data_ptr())


def _database_of(images, rows, seed, kind):
    """A database of `rows` rows, some of them near-duplicates of the images' hashes."""
    ctx, n = context(), images.shape[0]
    hashes = torch.empty((n * 8, 32), dtype=torch.uint8, device="cuda")
    yp.core.hash_batch_device(ctx, _ptr(images), n, KINDS[kind], d_hashes=_ptr(hashes))
    db = _synth_rows(rows, seed)
    _plant(db, hashes, max(4 * n, rows // 10_000), seed)
    torch.cuda.synchronize()
    rows = _Rows(db)
    return yp.Database(ctx, device_buffer=rows, n_rows=db.shape[0])


def prepare(case, seed):
    op, ctx = case["op"], context()
    if op == "hash":
        n = case["n"]
        images = _images(case["input"], n, seed)
        new = lambda shape, dt: torch.zeros(shape, dtype=dt, device="cuda")  # noqa: E731
        return {"op": op, "images": images, "n": n, "kind": KINDS[case["input"]],
                "dct": JAROSZ if case["filter"] == "jarosz" else yp._lib.DCT_FP32,
                "out": {"hashes": new((n, 8, 32), torch.uint8), "quality": new((n, 8), torch.float32),
                        "thresholds": new((n, 8), torch.float32), "pdqf": new((n, 256), torch.float32)}}
    if op == "match":
        queries = _synth_rows(case["queries"], seed + 1_000_003)
        rows = _synth_rows(case["rows"], seed)
        _plant(rows, queries, case["rows"] // 1000, seed)
        torch.cuda.synchronize()
        db = yp.Database(ctx, device_buffer=_Rows(rows), n_rows=case["rows"])
        return {"op": op, "matcher": yp.CudaMatcher(ctx, db, case["threshold"]),
                "needles": queries.cpu().numpy(), "found": np.zeros(1 << 15, yp.HIT_DTYPE)}
    if op == "scan":
        if case["clustered"]:
            rows, queries = _clustered(case["rows"], case["queries"], seed)
            capacity = case["queries"] * MEMBERS + 4096
        else:
            rows = _synth_rows(case["rows"], seed)
            queries = _synth_rows(case["queries"], seed + 1_000_003)
            _plant(rows, queries, case["rows"] // 1000, seed)
            capacity = 1 << 16
        torch.cuda.synchronize()
        return {"op": op, "rows": rows, "queries": queries, "threshold": case["threshold"],
                "hits": torch.zeros((capacity, 4), dtype=torch.int32, device="cuda"),
                "count": ctx.alloc(8)}
    if op == "screen":
        images = _images(case["input"], case["n"], seed)
        return {"op": op, "db": _database_of(images, case["rows"], seed, case["input"]),
                "images": _pinned(images), "threshold": case["threshold"],
                "found": np.zeros(1 << 13, yp.HIT_DTYPE)}
    rng = np.random.default_rng(seed)
    images = _images(case["input"], 256, seed)
    db = _database_of(images, case["rows"], seed, case["input"])
    count = np.exp(rng.uniform(0, math.log(64), case["requests"])).astype(np.uint32)
    server = yp.Server(ctx, db, threshold=case["threshold"], input_kind=case["input"],
                       max_step_images=256, step_hit_capacity=1 << 17)
    return {"op": op, "db": db, "server": server, "pool": _pinned(images), "count": count,
            "first": rng.integers(0, 256 - count, dtype=np.uint32)}


# --------------------------------------------------------------------------------- a pass

def run(state):
    op, ctx = state["op"], context()
    if op == "hash":
        out = state["out"]
        yp.core.hash_batch_device(ctx, _ptr(state["images"]), state["n"], state["kind"],
                                  _ptr(out["hashes"]), _ptr(out["quality"]), _ptr(out["thresholds"]),
                                  _ptr(out["pdqf"]), 1, None, state["dct"])
        return out
    if op == "match":
        return _kept(state["found"], state["matcher"].find_all(state["needles"]))
    if op == "scan":
        hits, rows, queries = state["hits"], state["rows"], state["queries"]
        yp.core.scan_device(ctx, _ptr(rows), rows.shape[0], _ptr(queries), queries.shape[0],
                            state["threshold"], _ptr(hits), hits.shape[0], state["count"])
        total = int(state["count"].download((1,), np.uint64)[0])
        yp.core.sort_hits_device(ctx, _ptr(hits), min(total, hits.shape[0]))
        return {"total": total, "hits": hits}
    if op == "screen":
        hits, hashes = yp.screen_host(ctx, state["db"], state["images"].array, state["threshold"],
                                      want_hashes=True)
        return dict(_kept(state["found"], hits), hashes=hashes)
    submitted, rejected, n_hits, hits = state["server"].replay(
        state["pool"].array, state["first"], state["count"], hit_capacity=4096)
    return {"submitted": submitted, "rejected": rejected, "n_hits": n_hits.view(np.int64),
            "hits": hits.view(np.int64)}


def _kept(found, hits):
    """The hits in the program's own list of records."""
    found[:len(hits)] = hits
    return {"total": len(hits), "hits": found.view(np.int64)}


def work(case):
    """Bytes: every input read once and every output written once. Operations: the DCT's and
    the compress's multiply-adds, an exclusive-or and a count per bit pair of a scan."""
    op = case["op"]
    if op == "hash":
        n = case["n"]
        ops = (512 * 512 * 8 if case["filter"] == "jarosz" else 2 * 27 * 127 * 127)
        return {"bytes": n * (IMAGE_BYTES[case["input"]] + 256 + 64 + 1024),
                "flops": n * (ops + 2 * 16 * 127 * 127 + 2 * 16 * 16 * 127)}
    if op in ("match", "scan"):
        q, rows = case["queries"], case["rows"]
        return {"bytes": 32 * (q + rows), "flops": 2 * 256 * q * rows}
    if op == "screen":
        n = case["n"]
        return {"bytes": n * (IMAGE_BYTES[case["input"]] + 256) + 32 * case["rows"],
                "flops": 2 * 256 * 8 * n * case["rows"]}
    images = int(case["requests"] * 63 / math.log(64))  # the mean of a log-uniform 1..64
    return {"bytes": images * IMAGE_BYTES[case["input"]] + 32 * case["rows"],
            "flops": 2 * 256 * 8 * images * case["rows"]}


# ---------------------------------------------------------------------- values in 64 bits

def _tent_matrix():
    """[127, 512]: row o holds the weights (1, 2, 3, 2, 1) / 9 at columns 4 o + 2 .. 4 o + 6
    (the 2-D filter is their outer product, k / 81)."""
    m = torch.zeros((127, 512), dtype=torch.float64, device="cuda")
    for o in range(127):
        m[o, 4 * o + 2:4 * o + 7] = torch.tensor([1, 2, 3, 2, 1], dtype=torch.float64) / 9
    return m


def _box_matrix():
    """[127, 512]: two box filters of window 3 (2 at the ends of a line), then the samples
    at ((2 o + 1) 512) / 254."""
    box = torch.zeros((512, 512), dtype=torch.float64, device="cuda")
    for i in range(512):
        lo, hi = max(0, i - 1), min(511, i + 1)
        box[i, lo:hi + 1] = 1.0 / (hi - lo + 1)
    return (box @ box)[[((2 * o + 1) * 512) // 254 for o in range(127)]]


def _luma64(images, kind):
    x = images.double()
    if kind in ("rgb8", "rgba8"):
        x = 0.299 * x[..., 0] + 0.587 * x[..., 1] + 0.114 * x[..., 2]
    return x


def exact(case, seed):
    if case["op"] != "hash":
        return None  # hits and hashes are whole numbers
    n = case["n"]
    images = _images(case["input"], n, seed)
    filt = _box_matrix() if case["filter"] == "jarosz" else _tent_matrix()
    k = torch.arange(1, 17, dtype=torch.float64, device="cuda")[:, None]
    i = torch.arange(127, dtype=torch.float64, device="cuda")[None]
    dct = math.sqrt(2 / 127) * torch.cos(math.pi * k * (2 * i + 1) / 254)
    left = dct @ filt
    pdqf = torch.cat([left @ _luma64(images[s:s + 64], case["input"]) @ left.T
                      for s in range(0, n, 64)])
    # slots 0-3: the sign of every other row and column; slots 4-7: their transposes, in the
    # order of the library's outputs. Thresholds are the 128th smallest values of slots 0-3.
    sign = torch.ones(16, dtype=torch.float64, device="cuda")
    sign[0::2] = -1
    r, c = sign[:, None], sign[None, :]
    flips = [1, c, r * c, r]
    thr = torch.stack([(pdqf * f).reshape(n, 256).sort(1).values[:, 127] for f in flips], 1)
    slots = [pdqf * f for f in flips]
    t = pdqf.transpose(1, 2)
    slots += [t, t * r, t * (r * c), t * c]
    quality = torch.stack([((s[:, 1:] - s[:, :-1]).abs().sum((1, 2)) +
                            (s[:, :, 1:] - s[:, :, :-1]).abs().sum((1, 2))) / 180 for s in slots], 1)
    return {"hashes": None, "quality": quality.clamp(max=1.0),
            "thresholds": torch.cat([thr, thr], 1), "pdqf": pdqf.reshape(n, 256)}

