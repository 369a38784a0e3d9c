"""Sub-blocks of at most 32 chains in a relay of the four decision warps,
against the same sweeps with the sub-blocks of one warp (larger work items,
folds 1 and 2) and against the oracle (fold 4, where every item has at most 32
chains, and the smallest and fullest items of every fold).

The two forms add the same corrections in the same order, so states, energies
and slots are compared bit for bit, also with couplings that are not exact.
"""
import numpy as np
import pytest

from test_gpu_small import _compare, _geometric, _problem

pytestmark = pytest.mark.gpu


@pytest.fixture
def sequential_mode():
    from pysa_gb300 import _lib
    lib = _lib.load()
    _lib.check(lib.pysa_gb_set_decision_mode(2), "mode")
    yield
    _lib.check(lib.pysa_gb_set_decision_mode(0), "mode reset")


def _run(J, h, ptype, R, reads, update, item_chains, sweeps):
    from pysa_gb300 import Instance, PTBatch, pack_spins
    b = PTBatch(ptype, [Instance(J, h, _geometric(R), reads)], kernel="tc")
    b._setup_tc(64, item_chains=item_chains)
    x = np.random.default_rng(5).choice(
        [-1.0, 1.0] if ptype == "ising" else [0.0, 1.0],
        size=(R * reads, len(h))).astype(np.float32)
    b.set_states(pack_spins(x, ptype, b.words))
    b.run(sweeps, seed=11, update=update)
    return b.fetch()


@pytest.mark.parametrize("update", ["sequential", "random"])
@pytest.mark.parametrize("n,wide", [
    (64, 128), (79, 128), (300, 64), (512, 128), (513, 64), (700, 64),
    (1024, 64)])
def test_relay_equals_one_warp(sequential_mode, n, wide, update):
    rng = np.random.default_rng(n)
    J = np.triu(rng.normal(size=(n, n)) / np.sqrt(n), 1).astype(np.float32)
    J = J + J.T
    h = rng.normal(size=n).astype(np.float32)
    a = _run(J, h, "ising", 8, 16, update, 32, 6)
    b = _run(J, h, "ising", 8, 16, update, wide, 6)
    for k in a:
        assert np.array_equal(a[k], b[k]), k


@pytest.mark.parametrize("update", ["sequential", "random"])
@pytest.mark.parametrize("n,R,Rd", [
    (65, 1, 1), (127, 32, 2), (128, 31, 1), (577, 5, 1), (640, 32, 1),
    (1025, 32, 1), (1087, 3, 2), (1300, 16, 2)])
def test_relay_matches_oracle(oracle, sequential_mode, n, R, Rd, update):
    J, h = _problem(np.random.default_rng(n + R), n, True)
    _compare(oracle, "qubo", [(J, h)], [(R, Rd)], update,
             4 if n < 1000 else 2, _geometric)
