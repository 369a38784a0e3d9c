"""Fields and energies of sparse instances: fixed records and grouped rows,
couplings that span nine decades, sums outside the f32 range.

Oracle: the exactly rounded f64 sum (math.fsum) of the products, which are
exact.  The kernel's sums carry 72 bits, so a field is that sum rounded to f32
(half an f32 ulp, 2^-24, and 2^-40 for the double rounding) and an energy
likewise.
"""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _setup(J, h, x, ptype):
    from scipy.sparse import csr_matrix
    from pysa_gb300 import Instance, PTBatch, pack_spins
    b = PTBatch(ptype, [Instance(csr_matrix(J), h, np.ones(1, np.float32),
                                 len(x))], sparse=True)
    b.set_states(pack_spins(x, ptype, b.words))
    return (b.fields.cpu().numpy()[:len(x), :len(h)],
            b.energies.cpu().numpy()[:len(x)])


@pytest.mark.parametrize("ptype", ["ising", "qubo"])
@pytest.mark.parametrize("n,degree", [(1, 0), (40, 3), (300, 12), (257, 60),
                                      (700, 4)])
def test_sparse_fields_are_rounded_sums(ptype, n, degree):
    rng = np.random.default_rng(n)
    J = np.zeros((n, n), np.float32)
    for _ in range(n * degree // 2):
        i, j = rng.integers(n, size=2)
        if i != j:
            J[i, j] = J[j, i] = rng.normal() * 10.0 ** rng.uniform(-5, 4)
    h = rng.normal(size=n).astype(np.float32)
    x = rng.choice([-1.0, 1.0] if ptype == "ising" else [0.0, 1.0],
                   size=(5, n)).astype(np.float32)
    F, E = _setup(J, h, x, ptype)
    J64, h64, x64 = (a.astype(np.float64) for a in (J, h, x))
    for c in range(5):
        for i in range(n):
            want = math.fsum(np.append(J64[i] * x64[c], h64[i]))
            assert abs(F[c, i] - want) <= (2.0**-24 + 2.0**-40) * abs(want)
        want = math.fsum(np.append(
            (0.5 * J64 * x64[c][:, None] * x64[c][None]).ravel(), h64 * x64[c]))
        assert abs(E[c] - want) <= (2.0**-24 + 2.0**-40) * abs(want)


def test_sums_past_f32():
    n = 40
    J = np.zeros((n, n), np.float32)
    J[0, 1:] = J[1:, 0] = 3e38
    h = np.zeros(n, np.float32)
    x = np.ones((2, n), np.float32)
    x[1, 1::2] = -1.0  # its field and energy stay finite
    F, E = _setup(J, h, x, "ising")
    assert np.isinf(F[0, 0]) and np.isinf(E[0])
    want = math.fsum(J[0].astype(np.float64) * x[1])
    assert F[1, 0] == np.float32(want)
    assert E[1] == np.float32(want)
