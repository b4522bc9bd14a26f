"""Calls on a stream that is being captured are refused; the capture and the
context stay usable."""
import pytest
import torch

from housdorffhdf5cmake_gb300 import synth

pytestmark = pytest.mark.gpu

KEYS = ("hd", "hd_ab", "hd_ba", "sum_ab", "sum_ba", "n_a", "n_b", "status")


def _pair(shape):
    return synth.pair_from_spec(synth.PairSpec(shape, 3, "normal"), "cuda")


@pytest.mark.parametrize("metric", ["se6", "se18"])
@pytest.mark.parametrize("entry", ["compute", "compute_async", "compute_pipelined"])
@pytest.mark.parametrize("warm", [0, 1, 6])  # no workspace, one, one of every split group with results pending
def test_refused_call_leaves_the_capture(hd, ctx, entry, metric, warm):
    small, large = _pair((30, 70, 80)), _pair((60, 90, 130))  # the large one needs a larger workspace
    want = [ctx.compute(*p, metric) for p in (small, large)]
    x = torch.zeros(4, device="cuda")
    outs = [torch.empty(hd.RESULT_BYTES, dtype=torch.uint8, device="cuda") for _ in range(warm + 2)]
    stream = torch.cuda.Stream()
    torch.cuda.synchronize()
    with hd.Context(0) as c:
        def call(p, i):
            r = getattr(c, entry)(*p, metric, **({} if entry == "compute" else {"out": outs[i]}))
            return r if entry == "compute" else None

        with torch.cuda.stream(stream):
            for i in range(warm):
                call(small, i)
        torch.cuda.synchronize()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=stream, capture_error_mode="thread_local"):
            x.add_(1)
            for p in (small, large):
                with pytest.raises(hd.HDError):
                    call(p, warm)
        g.replay()
        torch.cuda.synchronize()
        assert x.tolist() == [1.0] * 4
        with torch.cuda.stream(stream):
            got = [call(p, warm + i) for i, p in enumerate((small, large))]
            if entry == "compute_pipelined":
                c.flush()
        torch.cuda.synchronize()
        if entry != "compute":
            got = [hd.result_from_bytes(o.cpu()) for o in outs]
            want = [want[0]] * (warm + 1) + [want[1]]
        for i, (a, b) in enumerate(zip(got, want)):
            assert all(a[k] == b[k] for k in KEYS), (i, a, b)
