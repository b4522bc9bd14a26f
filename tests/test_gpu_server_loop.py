"""The server where its groups (the distance transform) do not solve every
request: requests that only the dilation loop can take among ones that groups
take, and servers whose element or options ask for the loop.  A result whose
`iterations` is not 0 came from the loop."""
import json
import time

import numpy as np
import pytest
import torch

from housdorffhdf5cmake_gb300 import synth

pytestmark = pytest.mark.gpu

KEYS = ("hd", "hd_ab", "hd_ba", "hd_robust", "sum_ab", "sum_ba", "n_a", "n_b", "n_a_not_b", "n_b_not_a", "status")


def same(x, y):
    return all(x[k] == y[k] for k in KEYS)


def _pairs(n, seed, lo, hi, edge=0.0):
    return [synth.pair_from_spec(s, "cuda") for s in synth.batch_ragged_specs(seed, n=n, lo=lo, hi=hi, edge_frac=edge)]


@pytest.mark.parametrize("shape,budget", [((256, 256, 256), 24 << 20),  # 17 MB in the loop, 38 MB in a group
                                          ((8, 513, 40), 0)])           # beyond the transform's sizes
def test_request_for_the_loop_before_many_others(hd, ctx, shape, budget):
    """A request that no group can take is solved while requests submitted after it
    still wait, though those come faster than the groups take them."""
    big = synth.pair_from_spec(synth.PairSpec(shape, 3, "normal"), "cuda")
    others = _pairs(4, 61, 150, 170)
    want_big, want = ctx.compute(*big, "se6"), [ctx.compute(*p, "se6") for p in others]
    before, after = 50, 800
    with hd.Server(ctx, hbm_budget_bytes=budget) as srv:
        kind = {}
        for i in range(before + after):
            if i == before:
                t_big = srv.submit(*big)
            kind[srv.submit(*others[i % len(others)])] = i % len(others)
        at = None
        for i in range(before + after + 1):
            t, r = srv.wait_any(60000)
            if t == t_big:
                at = i
            assert same(r, want_big if t == t_big else want[kind[t]]), i
        st = srv.stats()
    assert at < before + after // 2, at
    assert not budget or st["bytes_peak"] <= budget


def test_resident_pair_among_steady_others(hd, ctx):
    """A pair of 64 barrier iterations that only the loop takes is done before most
    of the requests that arrive at a steady 38 k a second and are solved in groups."""
    far = synth.pair_far_blobs(5, (200, 513, 300), "cuda", min_dist=80.0)
    others = _pairs(8, 63, 190, 210)
    want_far, want = ctx.compute(*far, "se6"), [ctx.compute(*p, "se6") for p in others]
    n, pace = 4000, 26e-6
    with hd.Server(ctx, max_queue=2 * n) as srv:
        kind, at, t0 = {}, None, time.perf_counter()
        for i in range(n):
            while time.perf_counter() - t0 < i * pace:
                pass
            if i == 200:
                t_far = srv.submit(*far)
            kind[srv.submit(*others[i % 8])] = i % 8
        for i in range(n + 1):
            t, r = srv.wait_any(60000)
            if t == t_far:
                at = i
            assert same(r, want_far if t == t_far else want[kind[t]]), i
    assert at < n // 3, at


LOOP = [("se18", {}), ("se6", {"kernel": 2})]


def _from_loop(r):
    return r["iterations"] > 0 or r["hd"] <= 0


@pytest.mark.parametrize("metric,opts", LOOP)
def test_lone_request_then_burst(hd, metric, opts):
    """A long lone request, then a burst that fills the two slots and queues up
    behind: the server drains and goes on in its other brick shape, and the lone
    request after the burst has the first shape again."""
    lone = synth.pair_far_blobs(3, (192, 192, 192), "cuda", min_dist=75.0)
    burst = _pairs(30, 41, 32, 96, edge=0.1)
    with hd.Context(0, **opts) as c:
        want_lone, want = c.compute(*lone, metric), [c.compute(*p, metric) for p in burst]
        with hd.Server(c, metric=metric, max_inflight=2) as srv:
            for _ in range(3):
                t0 = srv.submit(*lone)
                ts = [srv.submit(*p) for p in burst]
                res = [srv.wait(t, 60000) for t in ts] + [srv.wait(t0, 60000)]
                for i, (r, w) in enumerate(zip(res, want + [want_lone])):
                    assert same(r, w) and _from_loop(r), i
                r = srv.wait(srv.submit(*lone), 60000)
                assert same(r, want_lone) and _from_loop(r)


@pytest.mark.parametrize("metric,opts", LOOP)
def test_cancel_in_the_loop(hd, metric, opts):
    """A pair cancelled while it dilates leaves the loop; pairs beside it and pairs
    that take its slot afterwards get their own results."""
    far = synth.pair_far_blobs(5, (512, 512, 512), "cuda")
    pairs = _pairs(6, 43, 64, 128)
    with hd.Context(0, **opts) as c:
        want = [c.compute(*p, metric) for p in pairs]
        with hd.Server(c, metric=metric, tick_iterations=1, max_inflight=3) as srv:
            for _ in range(2):
                tf = srv.submit(*far)
                t0 = time.time()
                while srv.stats()["resident_pairs"] == 0 and time.time() - t0 < 10:
                    pass
                ts = [srv.submit(*p) for p in pairs[:2]]
                srv.cancel(tf)
                ts += [srv.submit(*p) for p in pairs[2:]]
                assert srv.wait(tf, 60000)["status"] == hd.HD_ERR_CANCELLED
                for i, t in enumerate(ts):
                    r = srv.wait(t, 60000)
                    assert same(r, want[i]) and _from_loop(r), i
            st = srv.stats()
    assert st["cancelled"] == 2 and st["resident_pairs"] == st["waiting_pairs"] == 0


@pytest.mark.parametrize("metric,opts", LOOP)
def test_budget_and_mix_in_the_loop(hd, metric, opts):
    """Loop admission under a budget of a few pairs, an oversize request, and each
    result the same alone and in the mix."""
    pairs = _pairs(16, 13, 64, 96)
    budget = 24 << 20
    with hd.Context(0, **opts) as c:
        want = [c.compute(*p, metric) for p in pairs]
        with hd.Server(c, metric=metric, hbm_budget_bytes=budget, tick_iterations=2) as srv:
            for i in (0, 9):
                r = srv.wait(srv.submit(*pairs[i]), 60000)
                assert same(r, want[i]) and _from_loop(r)
            big = torch.zeros((320, 320, 320), dtype=torch.uint8, device="cuda")
            tbig = srv.submit(big, big)
            ts = [srv.submit(*p) for p in pairs]
            for i, t in enumerate(ts):
                r = srv.wait(t, 60000)
                assert same(r, want[i]) and _from_loop(r), i
            assert srv.wait(tbig, 60000)["status"] == hd.HD_ERR_OOM
            assert srv.stats()["bytes_peak"] <= budget


def test_groups_given_back_to_the_loop(hd, ctx, tmp_path):
    """A tuning table that names the dilation loop: every group is refused and its
    requests go to the loop."""
    entry = {"kernel": 2, "bxw": 4, "bz": 8, "steps": 2, "ctas_per_sm": 0, "order": 0, "spread": 0, "us": 1.0}
    table = tmp_path / "table.json"
    table.write_text(json.dumps({"version": 1, "entries": {f"se6/v{v}/{p}": entry for v in range(30)
                                                           for p in ("p1", "p2", "p16")}}))
    pairs = _pairs(24, 71, 24, 112, edge=0.2)
    host = [tuple(np.ascontiguousarray(m.cpu().numpy()) for m in p) for p in pairs]
    want = [ctx.compute(*p, "se6") for p in pairs]
    with hd.Context(0, tuning_table=str(table)) as c, hd.Server(c) as srv:
        ts = [srv.submit(*(h if i % 3 == 0 else p)) for i, (p, h) in enumerate(zip(pairs, host))]
        for i, t in enumerate(ts):
            r = srv.wait(t, 60000)
            assert same(r, want[i]) and _from_loop(r), i
