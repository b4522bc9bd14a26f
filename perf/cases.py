"""Performance cases of the Hausdorff-distance library: the calls a user's program makes.

Each case is one pass through a public entry point of the Python package on
seeded synthetic masks (``housdorffhdf5cmake_gb300.synth``), with the sizes,
structuring elements and entry points that the benchmark, the tests and the
command-line configurations of this repository use.  ``listed()`` are the
cases, ``draw()`` gives further ones of the same ranges.

The result field ``iterations`` (grid-barrier iterations of the device loop, a
diagnostic that the library documents as depending on the kernel shape) is
left out of the outputs; every other field is returned.
"""
import math

import numpy as np
import torch

import housdorffhdf5cmake_gb300 as hd
from housdorffhdf5cmake_gb300 import synth

INTS = ("hd", "hd_ab", "hd_ba", "hd_robust", "sum_ab", "sum_ba", "n_a", "n_b", "n_a_not_b", "n_b_not_a", "status")
PERCENTILE = 0.95  # the library's default

_contexts = {}
_servers = {}


def _context(label=0):
    """A program keeps one context per label it looks at."""
    if label not in _contexts:
        _contexts[label] = hd.Context(0, label=label)
    return _contexts[label]


def _server(metric):
    if metric not in _servers:
        _servers[metric] = hd.Server(hd.Context(0), metric=metric)
    return _servers[metric]


def listed():
    return [
        # one small structure per mask: the latency of a lone blocking call
        {"name": "small_64", "entry": "compute", "masks": "salt", "metric": "se6", "W": 64, "H": 64, "D": 64},
        # a crop around a lesion, odd sizes, under the drop-in's default element
        {"name": "crop_odd_se18", "entry": "compute", "masks": "union", "metric": "se18", "W": 117, "H": 131, "D": 75},
        # a CT-like pair (segmentation against ground truth), blocking
        {"name": "ct_se6", "entry": "compute", "masks": "union", "metric": "se6", "W": 512, "H": 512, "D": 256},
        # the same under the reference's shipped element
        {"name": "ct_se18", "entry": "compute", "masks": "union", "metric": "se18", "W": 512, "H": 512, "D": 256},
        # evaluation loop over device-resident CT pairs: enqueued back to back, one flush
        {"name": "ct_pipelined_8", "entry": "pipelined", "masks": "union", "metric": "se6", "W": 512, "H": 512,
         "D": 256, "pairs": 8},
        # one structure of uint8 label volumes of an odd size, enqueued on the caller's stream
        {"name": "label_async_6", "entry": "async", "masks": "label", "metric": "se6", "W": 301, "H": 287, "D": 173,
         "pairs": 6, "label": 3},
        # few small blobs far apart: hundreds of dilation steps
        {"name": "far_blobs_512", "entry": "compute", "masks": "blobs", "metric": "se6", "W": 512, "H": 512, "D": 512},
        # host masks (pinned), the reference's own way in
        {"name": "host_ct_se18", "entry": "host", "masks": "union", "metric": "se18", "W": 512, "H": 512, "D": 256},
        # a test set in one call: ragged shapes, empty and identical masks among them
        {"name": "batch_256", "entry": "batch", "masks": "ragged", "metric": "se6", "lo": 64, "hi": 384, "pairs": 256},
        # patches of a training loop's validation step under the shipped element
        {"name": "batch_patches_se18", "entry": "batch", "masks": "ragged", "metric": "se18", "lo": 24, "hi": 96,
         "pairs": 48},
        # per-voxel distance maps of one pair (error display)
        {"name": "map_256", "entry": "map", "masks": "union", "metric": "se6", "W": 256, "H": 256, "D": 160},
        # a burst of requests of mixed sizes through the server
        {"name": "server_24", "entry": "server", "masks": "stream", "metric": "se6", "pairs": 24},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    entry = rng.choice(["compute", "compute", "compute", "pipelined", "async", "host", "batch", "batch", "map",
                        "server"])
    metric = rng.choice(["se6", "se6", "se18"])
    if entry == "batch":
        lo = _log(rng, 16, 64)
        hi = _log(rng, max(80, lo + 8), 384)
        return {"entry": "batch", "masks": "ragged", "metric": metric, "lo": lo, "hi": hi,
                "pairs": _log(rng, 2, 256 if hi < 256 else 96)}
    if entry == "server":
        return {"entry": "server", "masks": "stream", "metric": metric, "pairs": _log(rng, 1, 24)}
    case = {"entry": entry, "metric": metric, "W": _log(rng, 40, 512), "H": _log(rng, 40, 512), "D": _log(rng, 24, 400)}
    case["masks"] = rng.choice(["union", "union", "salt"])
    if entry == "compute" and rng.random() < 0.25:
        # the blobs' distance scales with the smallest axis, 200 voxels at 512
        case.update(masks="blobs", W=_log(rng, 256, 512), H=_log(rng, 256, 512), D=_log(rng, 256, 480))
    if entry == "async":
        case.update(masks="label", label=rng.randint(1, 5))
    if entry in ("pipelined", "async"):
        case["pairs"] = rng.randint(2, 8)
    return case


def _pair(case, seed, device):
    """One pair of masks of a case, (D, H, W) uint8."""
    shape = (case["D"], case["H"], case["W"])
    kind = case["masks"]
    if kind == "salt":
        return synth.pair_ellipsoid_salt(seed, shape, device)
    if kind == "blobs":
        return synth.pair_far_blobs(seed, shape, device, min_dist=200.0 * min(shape) / 512)
    a, b = synth.pair_from_spec(synth.PairSpec(shape, seed, "normal"), device)
    if kind == "label":
        # the structure under its label, another one beside it, background 0
        lab = case["label"]
        other = 1 + (lab % 5)
        a, b = (torch.where(m != 0, lab, other * torch.roll(m, m.shape[2] // 3, 2)).to(torch.uint8) for m in (a, b))
    return a, b


def _pairs(case, seed, device):
    kind = case["masks"]
    seed = seed % (1 << 20)  # the generators multiply a pair's seed within 64 bits
    if kind == "ragged":
        specs = synth.batch_ragged_specs(seed, n=case["pairs"], lo=case["lo"], hi=case["hi"])
        return [synth.pair_from_spec(synth.PairSpec(s.shape, seed * 256 + i, s.kind), device)
                for i, s in enumerate(specs)]
    if kind == "stream":
        reqs = synth.serving_stream(seed, case["pairs"], 0.0)
        return [synth.pair_from_spec(synth.PairSpec(r.shape, seed * 256 + i, "normal"), device)
                for i, r in enumerate(reqs)]
    return [_pair(case, seed * 256 + i, device) for i in range(case.get("pairs", 1))]


def _columns(raw):
    """The fields of a block of result records (bytes on the device), as views."""
    i32, i64, f64 = raw.view(torch.int32), raw.view(torch.int64), raw.view(torch.float64)
    return {"hd": i32[:, 0], "sums_counts": i64[:, 1:7], "avg_hd": f64[:, 7], "status_hds": i32[:, 16:20]}


def prepare(case, seed):
    entry = case["entry"]
    st = {"entry": entry, "metric": case["metric"]}
    pairs = _pairs(case, seed, "cuda")
    if entry == "host":
        pairs = [(a.cpu().pin_memory(), b.cpu().pin_memory()) for a, b in pairs]
    st["pairs"] = pairs
    if entry == "server":
        st["server"] = _server(case["metric"])
        torch.cuda.synchronize()
        return st
    ctx = st["ctx"] = _context(case.get("label", 0))
    if entry in ("pipelined", "async"):
        raw = torch.zeros((len(pairs), hd.RESULT_BYTES), dtype=torch.uint8, device="cuda")
        st["raw"], st["columns"] = list(raw), _columns(raw)
    elif entry == "batch":
        st["batch"] = ctx.prepare_batch(pairs, case["metric"])
    torch.cuda.synchronize()
    return st


def _fields(r):
    out = {k: r[k] for k in INTS}
    out["avg_hd"] = r["avg_hd"]
    return out


def run(st):
    entry, metric = st["entry"], st["metric"]
    if entry in ("compute", "host"):
        (a, b), = st["pairs"]
        return _fields(st["ctx"].compute(a, b, metric))
    if entry == "pipelined":
        ctx = st["ctx"]
        for (a, b), out in zip(st["pairs"], st["raw"]):
            ctx.compute_pipelined(a, b, metric, out=out)
        ctx.flush()
        return st["columns"]
    if entry == "async":
        ctx = st["ctx"]
        for (a, b), out in zip(st["pairs"], st["raw"]):
            ctx.compute_async(a, b, metric, out=out)
        return st["columns"]
    if entry == "batch":
        cols = st["batch"].run(columns=True)
        cols.pop("iterations")
        return {k: v.view(np.int64) if v.dtype == np.uint64 else v for k, v in cols.items()}
    if entry == "map":
        (a, b), = st["pairs"]
        r, ma, mb = st["ctx"].distance_map(a, b, metric)
        return {"result": _fields(r), "map_a": ma, "map_b": mb}
    srv = st["server"]
    tickets = [srv.submit(a, b) for a, b in st["pairs"]]
    results = [_fields(srv.wait(t)) for t in tickets]
    return {k: np.array([r[k] for r in results]) for k in INTS + ("avg_hd",)}


def _voxels(case):
    """Voxels of one mask, summed over the pairs (the mean of the range for ragged shapes)."""
    kind = case["masks"]
    if kind == "ragged":
        return case["pairs"] * ((case["lo"] + case["hi"]) / 2) ** 3
    if kind == "stream":
        # log-normal scale (sigma 0.35) on 256 x 256 x 160 voxels, a tenth at 512^3
        return case["pairs"] * (0.9 * 256 * 256 * 160 * math.exp(0.5 * (3 * 0.35) ** 2) + 0.1 * 512 ** 3)
    return case.get("pairs", 1) * case["W"] * case["H"] * case["D"]


def work(case):
    """Both masks read once, the result records (and the int32 maps) written once."""
    n = _voxels(case)
    out = case.get("pairs", 1) * hd.RESULT_BYTES + (8 * n if case["entry"] == "map" else 0)
    return {"bytes": 2 * n + out, "flops": 0}


# ---- exact results, plain torch ---------------------------------------------
def _shift_or(dst, src, dz, dy, dx):
    D, H, W = src.shape

    def span(n, k):
        return slice(max(0, k), min(n, n + k)), slice(max(0, -k), min(n, n - k))

    (tz, fz), (ty, fy), (tx, fx) = span(D, dz), span(H, dy), span(W, dx)
    dst[tz, ty, tx] |= src[fz, fy, fx]


_FACES = [(1, 0, 0), (-1, 0, 0), (0, 1, 0), (0, -1, 0), (0, 0, 1), (0, 0, -1)]
_MORE = [(0, y, x) for y in (-1, 1) for x in (-1, 1)] + [(z, y, x) for z in (-1, 1) for y in (-1, 1) for x in (-1, 1)]


def _one_sided(src, tgt, offsets, want_map):
    """Steps at which the dilation of src first covers each voxel of tgt: histogram (index = step) and map."""
    left = tgt & ~src
    hist, cur, step = [0], src, 0
    dist = torch.where(tgt & src, 0, -1).to(torch.int32) if want_map else None
    total = int(left.sum())
    while total:
        step += 1
        nxt = cur.clone()
        for o in offsets:
            _shift_or(nxt, cur, *o)
        cur = nxt
        hit = left & cur
        n = int(hit.sum())
        hist.append(n)
        total -= n
        left &= ~cur
        if want_map:
            dist[hit] = step
    return np.array(hist, dtype=np.int64), dist


def _robust(hist, total):
    """First step k at which the share of covered voxels no longer lies under the percentile (float32 rule)."""
    bound = np.float32(total) * np.float32(PERCENTILE)
    return int(np.nonzero(~(bound > np.cumsum(hist).astype(np.float32)))[0][0])


def _exact_pair(a, b, metric, want_map=False):
    na, nb, nab = int(a.sum()), int(b.sum()), int((a & b).sum())
    r = dict.fromkeys(INTS, 0)
    r.update(n_a=na, n_b=nb, n_a_not_b=na - nab, n_b_not_a=nb - nab, avg_hd=0.0)
    if not na and not nb:
        return r, None, None
    if not na or not nb:
        r.update(hd=-1, hd_ab=-1, hd_ba=-1, hd_robust=-1, status=hd.HD_EMPTY_MASK, avg_hd=math.nan)
        return r, None, None
    offsets = _FACES + (_MORE if metric == "se18" else [])
    hab, ma = _one_sided(b, a, offsets, want_map)
    hba, mb = _one_sided(a, b, offsets, want_map)
    k = np.arange(max(len(hab), len(hba)), dtype=np.int64)
    r.update(hd_ab=len(hab) - 1, hd_ba=len(hba) - 1, hd=max(len(hab), len(hba)) - 1,
             sum_ab=int((k[:len(hab)] * hab).sum()), sum_ba=int((k[:len(hba)] * hba).sum()),
             hd_robust=max(_robust(hab, na - nab), _robust(hba, nb - nab)))
    r["avg_hd"] = float(r["sum_ab"] + r["sum_ba"]) / float(na + nb)
    return r, ma, mb


def exact(case, seed):
    if _voxels(case) > 3.5e9:
        return None
    lab = case.get("label", 0)
    rows = []
    for a, b in _pairs(case, seed, "cuda"):
        a, b = (a == lab, b == lab) if lab else (a != 0, b != 0)
        r, ma, mb = _exact_pair(a, b, case["metric"], case["entry"] == "map")
        rows.append(r)
    entry = case["entry"]
    if entry in ("compute", "host"):
        return rows[0]
    if entry == "map":
        return {"result": rows[0], "map_a": ma, "map_b": mb}
    col = {k: np.array([r[k] for r in rows]) for k in INTS + ("avg_hd",)}
    if entry in ("pipelined", "async"):
        return {"hd": col["hd"].astype(np.int32),
                "sums_counts": np.stack([col[k] for k in ("sum_ab", "sum_ba", "n_a", "n_b", "n_a_not_b", "n_b_not_a")],
                                        axis=1),
                "avg_hd": col["avg_hd"],
                "status_hds": np.stack([col[k] for k in ("status", "hd_ab", "hd_ba", "hd_robust")],
                                       axis=1).astype(np.int32)}
    return col
