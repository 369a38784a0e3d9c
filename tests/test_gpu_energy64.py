"""f64 energies from the problem tables: the edges of a 32-column, 128-row unit,
of the 1024 rows staged at a time, of the clusters and of the four states a
cluster takes; couplings that span nine decades; sums outside the f32 range.

Oracle: the exactly rounded sum (math.fsum) of the f64 products, which are
exact.  The kernel's sums carry 72 bits of their largest term until they are
converted with three f64 roundings, so it can lose 3 * 2^-53 of the result and,
over the n^2 additions to a triple's third part, n^2 2^-72 of S =
sum |J_ij| / 2 + |h_i|: below 2^-51 of S together.
"""
import ctypes
import math

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _energies(ptype, J, h, words, count):
    from pysa_gb300 import Instance, PTBatch
    from pysa_gb300._lib import check, ref
    b = PTBatch(ptype, [Instance(J, h, np.ones(1, np.float32), 1)],
                kernel="auto" if len(h) > 1 else "plain")
    w = torch.from_numpy(words.view(np.int32)).cuda()
    out = torch.full((count,), -7.0, dtype=torch.float64, device="cuda")
    check(b.lib.pysa_gb_energy64_tables(
        ref(b.p), ref(b._ht), 0, w.data_ptr(), words.shape[1], count,
        out.data_ptr(), torch.cuda.current_stream().cuda_stream), "energy64")
    torch.cuda.synchronize()
    return out.cpu().numpy()


def _case(rng, ptype, n, count, spread):
    from pysa_gb300 import pack_spins
    J = rng.normal(size=(n, n))
    if spread:
        J *= 10.0 ** rng.uniform(-5, 4, size=(n, n))
    J = np.triu(J, 1)
    J = (J + J.T).astype(np.float32)
    h = rng.normal(size=n).astype(np.float32)
    x = rng.choice([-1.0, 1.0] if ptype == "ising" else [0.0, 1.0],
                   size=(count, n)).astype(np.float32)
    return J, h, x, pack_spins(x, ptype, (n + 31) // 32)


@pytest.mark.parametrize("ptype", ["ising", "qubo"])
@pytest.mark.parametrize("n,count,spread", [
    (1, 1, False), (31, 3, False), (33, 5, True), (128, 4, True),
    (161, 2, False), (260, 9, True), (1024, 1, True), (1025, 6, False),
    (1100, 3, True)])
def test_energies_to_the_last_bits(ptype, n, count, spread):
    rng = np.random.default_rng(n + count)
    J, h, x, words = _case(rng, ptype, n, count, spread)
    got = _energies(ptype, J, h, words, count)
    J64, h64 = J.astype(np.float64), h.astype(np.float64)
    for c in range(count):
        s = x[c].astype(np.float64)
        terms = (0.5 * J64 * s[:, None] * s[None, :]).ravel()
        want = math.fsum(np.concatenate([terms, h64 * s]))
        S = 0.5 * np.abs(J64).sum() + np.abs(h64).sum()
        assert abs(got[c] - want) <= 2.0**-51 * S


def test_sums_outside_the_f32_range():
    rng = np.random.default_rng(1)
    for ptype in ("ising", "qubo"):
        J, h, x, words = _case(rng, ptype, 70, 5, False)
        x[1] = 1.0  # (numbers below: the aligned state leaves the range)
        J[:], h[3] = 0.0, 1.5
        J[0, 1:] = J[1:, 0] = 3e38
        from pysa_gb300 import pack_spins
        words = pack_spins(x, ptype, 3)
        got = _energies(ptype, J, h, words, 5)
        s = x.astype(np.float64)
        want = np.einsum("ci,ij,cj->c", s, J.astype(np.float64), s) / 2 + s @ h
        assert np.isfinite(got).all()
        assert np.abs(got - want).max() <= 2.0**-46 * 3e38 * 70
        J[0, 1] = J[1, 0] = np.inf  # a state of weight zero stays finite
        got = _energies(ptype, J, h, words, 5)
        assert not np.isfinite(got[1])
