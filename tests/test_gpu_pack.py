"""The packing kernel around the ends of its spans (128 words per warp, 16-byte
chunks): widths and base addresses at every alignment, one row to several
spans, masks of 0/1, of arbitrary nonzero bytes and of labels.  Counts and the
distances that follow from the packed words against the oracle: integers, no
tolerance."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def at_offset(m, off):
    """The mask as a CUDA tensor whose first byte lies `off` bytes past a 16-byte boundary, with foreground around it."""
    buf = torch.full((m.size + off + 16,), 3, dtype=torch.uint8, device="cuda")
    v = buf[off:off + m.size].view(m.shape)
    v.copy_(torch.from_numpy(m).cuda())
    assert v.data_ptr() % 16 == off
    return v


SHAPES = [(1, 1, 3), (3, 5, 7), (1, 1, 4095), (1, 1, 4096), (1, 2, 4097), (2, 64, 32), (2, 127, 31), (3, 43, 33),
          (1, 9, 447), (2, 17, 511), (5, 13, 301), (1, 129, 64)]


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("offs", [(0, 0), (1, 15), (8, 3)])
def test_span_ends(hd, ctx, oracle, shape, offs):
    rng = np.random.default_rng(sum(shape) + offs[0])
    a = (rng.random(shape) < 0.3).astype(np.uint8)
    b = (rng.random(shape) < 0.3).astype(np.uint8)
    a.flat[-1] = b.flat[0] = 1  # the first and last byte of a mask
    o = oracle.bfs_pair(a, b, "se6")
    with hd.Context(0, label=3) as lab:
        forms = [(ctx, a, b),
                 (ctx, a * rng.integers(1, 256, shape).astype(np.uint8), b * np.uint8(254)),
                 (lab, np.where(a != 0, 3, rng.integers(0, 3, shape)).astype(np.uint8),
                  np.where(b != 0, 3, rng.integers(4, 256, shape)).astype(np.uint8))]
        for c, ma, mb in forms:
            g = c.compute(at_offset(ma, offs[0]), at_offset(mb, offs[1]), "se6")
            for k in ("n_a", "n_b", "n_a_not_b", "n_b_not_a", "hd", "hd_ab", "hd_ba", "sum_ab", "sum_ba", "avg_hd"):
                assert g[k] == o[k], (k, g, o)


@pytest.mark.parametrize("shape", [(520, 512, 32), (311, 301, 96), (131, 257, 256)])
@pytest.mark.parametrize("label", [0, 3])
def test_pipelined_aligned_words(hd, ctx, shape, label):
    """The packing of the pipelined entry (rows of whole words, the next span asked
    for ahead: several spans per warp, a ragged end), with and without a label,
    against the blocking entry on masks of 0 and 1."""
    g = torch.Generator(device="cuda").manual_seed(sum(shape) + label)
    pairs, want = [], []
    for i in range(5):
        p = [torch.randint(0, 6, shape, generator=g, device="cuda", dtype=torch.uint8) for _ in range(2)]
        p[i % 2][i:] = 0
        p[i % 2].view(-1)[-1] = label or 1
        fg = [((m == label) if label else (m != 0)) for m in p]
        pairs.append(p)
        want.append(ctx.compute(*(m.to(torch.uint8) for m in fg), "se6"))
        assert (want[-1]["n_a"], want[-1]["n_b"]) == tuple(int(m.sum()) for m in fg)
    outs = [torch.empty(hd.RESULT_BYTES, dtype=torch.uint8, device="cuda") for _ in pairs]
    with hd.Context(0, label=label) as c:
        for p, o in zip(pairs, outs):
            c.compute_pipelined(*p, "se6", out=o)
        c.flush()
        torch.cuda.synchronize()
    for i, (o, w) in enumerate(zip(outs, want)):
        r = hd.result_from_bytes(o.cpu())
        assert all(r[k] == w[k] for k in r if k != "iterations"), (i, r, w)
