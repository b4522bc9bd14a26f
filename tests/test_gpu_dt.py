"""The distance-transform path (6-neighbour pairs by default) against
the dilation loop (a context that asks for it) and the oracle, on every field
but the barrier-loop count: sizes around its tiles (64 rows, 32 columns,
groups of 4 words, segments of 16 planes, 16 segments per CTA) and the limits
of the sizes it takes.  Integers: no tolerance."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

KEYS = ("hd", "hd_ab", "hd_ba", "hd_robust", "sum_ab", "sum_ba", "n_a", "n_b", "n_a_not_b", "n_b_not_a", "status",
        "avg_hd")


def same(g, w, tag):
    for k in KEYS:
        assert g[k] == w[k] or (k == "avg_hd" and g[k] != g[k] and w[k] != w[k]), (tag, k, g, w)


@pytest.fixture(scope="module")
def loop(hd):
    c = hd.Context(0, kernel=2)
    yield c
    c.close()


def masks(rng, shape, kind):
    a = np.zeros(shape, np.uint8)
    b = np.zeros(shape, np.uint8)
    D, H, W = shape
    if kind == "corners":  # the longest distance of the volume
        a[0, 0, 0] = 1
        b[-1, -1, -1] = 1
    elif kind == "sparse":
        for m in (a, b):
            for _ in range(3):
                m[rng.integers(D), rng.integers(H), rng.integers(W)] = 1
    elif kind == "slabs":  # empty planes and rows in between
        a[0] = 1
        b[:, H // 2, :] = 1
        b[-1, :, W // 3] = 1
    else:
        a[...] = rng.random(shape) < 0.03
        b[...] = rng.random(shape) < 0.01
        a[D // 2, H // 2, W // 2] = b[D // 3, H // 3, W // 3] = 1
    return a, b


SHAPES = [(1, 1, 1), (15, 31, 33), (16, 32, 32), (17, 33, 31), (2, 63, 127), (3, 64, 128), (5, 65, 129), (33, 4, 161),
          (31, 5, 96), (65, 127, 40), (8, 129, 260), (128, 3, 64), (129, 9, 30), (255, 7, 40), (256, 6, 33),
          (257, 5, 65), (300, 66, 20), (3, 511, 40), (2, 512, 70), (9, 449, 33), (4, 3, 2048), (1024, 4, 33)]


@pytest.mark.parametrize("shape", SHAPES)
def test_tile_edges(hd, ctx, loop, oracle, shape):
    rng = np.random.default_rng(sum(shape))
    for kind in ("corners", "sparse", "slabs", "random"):
        a, b = masks(rng, shape, kind)
        da, db = torch.from_numpy(a).cuda(), torch.from_numpy(b).cuda()
        g = ctx.compute(da, db, "se6")
        same(g, loop.compute(da, db, "se6"), (shape, kind))
        if a.size <= 70000:
            same(g, {**oracle.bfs_pair(a, b, "se6"), "hd_robust": g["hd_robust"]}, (shape, kind, "oracle"))


@pytest.mark.parametrize("shape", [(2, 513, 33), (1025, 3, 32), (2, 3, 2049)])
def test_sizes_beyond_its_limits_take_the_loop(hd, ctx, loop, shape):
    a, b = (torch.from_numpy(m).cuda() for m in masks(np.random.default_rng(1), shape, "corners"))
    with hd.Context(0, record_timings=True) as c:
        same(c.compute(a, b, "se6"), loop.compute(a, b, "se6"), shape)
        assert c.last_timings()["kernel"] == 2


def test_options_that_ask_for_the_loop(hd):
    a, b = (torch.from_numpy(m).cuda() for m in masks(np.random.default_rng(2), (20, 40, 70), "random"))
    for opts, kernel in (({}, 3), ({"kernel": 2}, 2), ({"brick_z": 8}, 2), ({"max_iterations": 500}, 2),
                         ({"ctas_per_sm": 1}, 2), ({"barrier_timeout_ns": 10**9}, 2), ({"steps_per_barrier": 2}, 2)):
        with hd.Context(0, record_timings=True, **opts) as c:
            c.compute(a, b, "se6")
            assert c.last_timings()["kernel"] == kernel, opts


@pytest.mark.parametrize("shape", [(17, 33, 70), (40, 66, 129), (257, 5, 33)])
def test_maps(hd, ctx, shape):
    rng = np.random.default_rng(3)
    with hd.Context(0, kernel=1) as one:
        for kind in ("sparse", "random"):
            a, b = (torch.from_numpy(m).cuda() for m in masks(rng, shape, kind))
            r, ma, mb = ctx.distance_map(a, b, "se6")
            w, wa, wb = one.distance_map(a, b, "se6")
            same(r, w, (shape, kind))
            assert torch.equal(ma, wa) and torch.equal(mb, wb)


def test_batches(hd, loop):
    """Groups of more pairs than one launch takes, of one pair each, more
    groups than workspaces, pairs without targets or sources; a pair beyond
    the limits takes the whole batch to the loop."""
    rng = np.random.default_rng(4)
    kinds = ("corners", "sparse", "slabs", "random")
    small = [masks(rng, s, k) for i, s in enumerate(SHAPES) for k in (kinds[i % 4], kinds[(i + 1) % 4])]
    z = np.zeros((9, 20, 50), np.uint8)
    one = z.copy()
    one[4, 5, 6] = 1
    small[3:3] = [(z, z), (z, one), (one, z), (one, one), (one, one | (rng.random(z.shape) < 0.1).astype(np.uint8))]
    large = [masks(rng, (200, 500, 500), "sparse") for _ in range(5)]
    with hd.Context(0, record_timings=True) as c:
        for tag, pairs, kernel in (("small", small, 3), ("mixed", small[:9] + large[:2] + small[9:20], 3),
                                   ("large", large, 3), ("two", small[8:10], 3),
                                   ("beyond", small[:3] + [masks(rng, (2, 513, 33), "sparse")], 2)):
            dev = [tuple(torch.from_numpy(m).cuda() for m in p) for p in pairs]
            got = c.batch(dev, "se6")
            assert c.last_timings()["kernel"] == kernel, tag
            for i, (g, p) in enumerate(zip(got, dev)):
                same(g, loop.compute(*p, "se6"), (tag, i))


@pytest.mark.parametrize("shape", [(1, 1, 3), (17, 33, 70), (3, 5, 1031)])
@pytest.mark.parametrize("offset,label", [(0, 0), (0, 3), (1, 0), (6, 3), (8, 0)])
def test_map_values_outside_the_transform(hd, shape, offset, label):
    """Maps of masks at any byte offset, with and without a label: -1 outside
    the mask, 0 on the overlap, at least 1 elsewhere."""
    rng = np.random.default_rng(6)
    n = int(np.prod(shape))
    flat = [torch.from_numpy(rng.integers(0, 5, n + offset, dtype=np.uint8)).cuda() for _ in range(2)]
    a, b = (f[offset:].view(shape) for f in flat)
    a.view(-1)[0] = b.view(-1)[-1] = label or 1
    fa, fb = ((m == label) if label else (m != 0) for m in (a, b))
    with hd.Context(0, label=label) as c:
        _, ma, mb = c.distance_map(a, b, "se6")
    for m, own, other in ((ma, fa, fb), (mb, fb, fa)):
        assert bool((m[~own] == -1).all()) and bool((m[own & other] == 0).all()) and bool((m[own & ~other] >= 1).all())


def test_groups_of_pairs_without_targets(hd, loop):
    """Full groups of identical, one-sided empty and empty masks, whose results are
    decoded (and whose counts are put back) where the columns are listed, with a
    few pairs that have columns between them, many times over."""
    rng = np.random.default_rng(7)
    pairs = []
    for i in range(128):
        a, b = masks(rng, SHAPES[1 + 7 * i % 15], ("random", "slabs")[i % 2])
        z = np.zeros_like(a)
        pairs.append(((a, a), (a, z), (z, b), (z, z), (b, b))[i % 5] if i % 16 else (a, b))
    dev = [tuple(torch.from_numpy(m).cuda() for m in p) for p in pairs]
    want = [loop.compute(*p, "se6") for p in dev]
    with hd.Context(0) as c:
        batch = c.prepare_batch(dev, "se6")
        for turn in range(50):
            for i, (g, w) in enumerate(zip(batch.run(), want)):
                same(g, w, (turn, i))


def test_tuning_table_of_several_entries(hd, loop, tmp_path):
    """Every entry of a table is read: workload classes with an entry of the loop
    take it, one whose entry names the transform and one without an entry do not."""
    rng = np.random.default_rng(8)
    entry = lambda kernel, steps: (f'{{"kernel": {kernel}, "bxw": 4, "bz": 8, "steps": {steps}, "ctas_per_sm": 0, '
                                   '"order": 0, "spread": 0, "us": 1.5}')
    table = {"se6/v12/p1": entry(2, 3), "se6/v15/p1": entry(1, 1), "se6/v15/p2": entry(2, 2), "se6/v18/p1": entry(3, 0)}
    path = tmp_path / "table.json"
    path.write_text('{\n  "version": 1,\n  "entries": {' + ",".join(f'\n    "{k}": {v}' for k, v in table.items()) +
                    "\n  }\n}\n")  # as the library writes it
    with hd.Context(0, tuning_table=str(path), record_timings=True) as c:
        for side, n, kernel, steps in ((16, 1, 2, 3), (32, 1, 1, 1), (32, 4, 2, 2), (64, 1, 3, 0), (64, 4, 3, 0)):
            a, b = (torch.from_numpy(m).cuda() for m in masks(rng, (side,) * 3, "random"))
            want = loop.compute(a, b, "se6")
            for g in [c.compute(a, b, "se6")] if n == 1 else c.batch([(a, b)] * n, "se6"):
                same(g, want, (side, n))
            t = c.last_timings()
            assert (t["kernel"], t["steps_per_barrier"]) == (kernel, steps), (side, n, t)


def test_no_memory_for_the_workspace(hd, ctx):
    """With room for the loop's workspace (1.6 GB) but not for the transform's (3.6
    GB): calls take the loop, and the autotuner measures the loop alone."""
    g = torch.Generator(device="cuda").manual_seed(5)
    pair = [(torch.rand((512, 512, 512), generator=g, device="cuda") < 0.01).to(torch.uint8) for _ in range(2)]
    want = ctx.compute(*pair, "se6")
    pairs = [pair] * 12
    torch.cuda.empty_cache()
    with hd.Context(0, record_timings=True) as c:
        c.compute(*(m[:8, :8, :8].contiguous() for m in pair), "se6")
        hog = torch.empty(torch.cuda.mem_get_info()[0] - (2600 << 20), dtype=torch.uint8, device="cuda")
        try:
            got = c.batch(pairs, "se6")
            timings = c.last_timings()
            report = c.autotune(pairs, "se6", repeats=1)
        finally:
            del hog
            torch.cuda.empty_cache()
        assert timings["kernel"] == 2 and "kernel=2" in report and "kernel=3" not in report
        for x in got:
            same(x, want, "loop")
        again = c.prepare_batch(pairs, "se6")
        assert again.run()[0]["sum_ab"] == want["sum_ab"]


def test_timings_name_no_loop(hd):
    """Timings of the transform: no iterations, no persistent grid, no bricks; of the
    loop: all of them."""
    a, b = (torch.from_numpy(m).cuda() for m in masks(np.random.default_rng(9), (40, 60, 70), "sparse"))
    out = torch.empty(hd.RESULT_BYTES, dtype=torch.uint8, device="cuda")
    fields = ("grid_ctas", "brick_x_words", "brick_z", "brick_rows", "steps_per_barrier")
    for opts in ({}, {"kernel": 2}):
        with hd.Context(0, record_timings=True, **opts) as c:
            def pipelined():
                c.compute_pipelined(a, b, "se6", out=out)
                c.flush()
                torch.cuda.synchronize()

            for call in (lambda: c.compute(a, b, "se6"), lambda: c.batch([(a, b)] * 3, "se6"), pipelined):
                call()
                t = c.last_timings()
                assert all((t[f] > 0) == bool(opts) for f in fields), (opts, t)
                assert t["kernel"] == opts.get("kernel", 3) and t["solve_ms"] > 0
