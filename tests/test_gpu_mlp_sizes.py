"""The proposal network's kernels at the edges of their tiles and split: one
and several 128-row batches, K of two 64-wide tiles (two stages in flight) and
more, layers of one and several column tiles, and buffers that are only 4-byte
aligned (scalar loads and stores).

Oracle: the same recipe in FP64 on BF16-rounded operands.  Products of BF16
values are exact in FP32 and sums of K <= 1024 of them err by at most K 2^-24
of the sum of their magnitudes; an operand that lands on the other side of a
BF16 boundary moves a result by 2^-8 of that term.  2e-3 of the largest value
covers both, as for the network's other comparisons.
"""
import numpy as np
import pytest
import torch

from oracle import mlp_oracle as mo

pytestmark = pytest.mark.gpu


def _err(got, want):
    return np.abs(got - want).max() / max(np.abs(want).max(), 1e-30)


@pytest.mark.parametrize("n,hidden,reads,offset", [
    (40, 256, 1, 0), (256, 512, 128, 0), (300, 256, 129, 0),
    (700, 1024, 20, 0), (100, 512, 200, 1)])
def test_network_at_tile_edges(n, hidden, reads, offset):
    from pysa_gb300 import Instance, PTBatch
    from pysa_gb300.proposal import LearnedProposal
    rng = np.random.default_rng(n + hidden)
    J = np.zeros((n, n), np.float32)
    inst = Instance(J, np.zeros(n, np.float32), np.ones(1, np.float32), reads)
    b = PTBatch("ising", [inst, inst])
    prop = LearnedProposal(b, hidden=hidden, lr=1e-2, init_seed=2)
    if offset:  # every FP32 buffer one float past a 16-byte boundary
        for k, t in list(prop.t.items()):
            if t.dtype == torch.float32:
                v = torch.zeros(t.numel() + 4, device=t.device)[1:1 + t.numel()]
                v = v.view(t.shape).copy_(t)
                prop.t[k] = v
                setattr(prop.m, k, v.data_ptr())
    I, B, nn, H = prop.I, prop.B, prop.nn, prop.H
    x = rng.choice([-1.0, 1.0], size=(I, B, nn)).astype(np.float32)
    tgt = (rng.random((I, B, nn)) < 0.2).astype(np.float32)
    rw = rng.random((I, B)).astype(np.float32)
    names = ("w1", "b1", "w2", "b2")
    w = {k: prop.t[k].cpu().numpy().astype(np.float64) for k in names}
    z2 = prop.forward(torch.from_numpy(x).cuda()).cpu().numpy()
    a1 = prop.t["a1"].cpu().numpy()
    prop.train_step(torch.from_numpy(tgt).cuda(), torch.from_numpy(rw).cuda())
    got = {k: prop.t[k].cpu().numpy() for k in prop.t if k != "pa"}
    for i in range(I):
        a1_o, z2_o = mo.forward(x[i], *(w[k][i] for k in names))
        assert _err(a1[i], a1_o) < 2e-3
        assert _err(z2[i], z2_o) < 2e-3
        # gradients from the GPU's own activations and logits
        p = 1 / (1 + np.exp(-z2[i].astype(np.float64)))
        dz2 = (rw[i] / rw[i].sum())[:, None] * (p - tgt[i])
        bf = lambda v: mo.bf16(np.asarray(v, np.float32)).astype(np.float64)
        da1 = (bf(got["dz2"][i]) @ bf(w["w2"][i])) * (a1[i] > 0)
        assert _err(got["dz2"][i], dz2) < 2e-3
        assert _err(got["da1"][i], da1) < 2e-3
        assert _err(got["dw2"][i], bf(got["dz2"][i]).T @ bf(a1[i])) < 2e-3
        assert _err(got["dw1"][i], bf(got["da1"][i]).T @ bf(x[i])) < 2e-3
        assert _err(got["db2"][i], got["dz2"][i].sum(0, dtype=np.float64)) < 2e-3
        assert _err(got["db1"][i], got["da1"][i].sum(0, dtype=np.float64)) < 2e-3
        for k in names:  # first Adam step: m / c1 = g, v / c2 = g^2
            g = got["d" + k][i].astype(np.float64)
            want = w[k][i] - 1e-2 * g / (np.abs(g) + 1e-8)
            big = np.abs(g) > 1e-6  # eps and f32 squares matter below
            assert np.abs(got[k][i] - want)[big].max() < 1e-5
    # the packed operands are the new weights: logits of the next forward
    z2 = prop.forward().cpu().numpy()
    for i in range(I):
        _, z2_o = mo.forward(x[i], *(got[k][i].astype(np.float64) for k in names))
        assert _err(z2[i], z2_o) < 2e-3
