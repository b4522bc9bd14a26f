"""The server where its groups (the distance transform) do not solve every
request: requests that only the dilation loop can take, among ones that groups
take."""
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
