"""The sparse-row sweep where its form changes: grouped rows (more than 32
neighbours) in 32-entry pieces, schedules made in order, sizes around the
smallest scheduled one, and more work items than SMs (narrow and wide schedules
then run in launches of their own)."""
import numpy as np
import pytest

from test_gpu_sparse_levels import _check, _graph

pytestmark = pytest.mark.gpu


def _problem(kind, n):
    rng = np.random.default_rng(n)
    if kind == "band":  # 40 neighbours each, in visiting order
        J = np.zeros((n, n), np.float32)
        for k in range(1, 21):
            i = np.arange(n - k)
            J[i, i + k] = rng.normal(size=n - k)
        J = (J + J.T).astype(np.float32)
    elif kind == "lattice":
        m = int(round(n ** 0.5))
        i = np.arange(n)
        J = np.zeros((n, n), np.float32)
        J[i, i // m * m + (i + 1) % m] = 1.0
        J[i, (i + m) % n] = 1.0
        J = np.triu(np.maximum(J, J.T), 1)
        J = (J + J.T).astype(np.float32)
    else:
        J = _graph(kind, n, rng)
    return J, rng.normal(size=n).astype(np.float32)


@pytest.mark.parametrize("update", ["sequential", "random"])
@pytest.mark.parametrize("kind,n,R,Rd", [
    ("ring", 32, 3, 1), ("ring", 33, 3, 1), ("ring", 64, 3, 1),
    ("ring", 65, 3, 1),                      # first scheduled sizes
    ("band", 130, 5, 2),                     # grouped rows, narrow
    (70, 400, 3, 1), (200, 420, 3, 1),       # rows of 2 and 5 pieces
    (24, 300, 4, 1), (12, 300, 4, 1),        # records of 32 and 16 in order
    ("ring", 900, 3, 1)])                    # a chunk past the round limit
def test_forms_match_oracle(oracle, kind, n, R, Rd, update):
    J, h = _problem(kind, n)
    for ptype in ("ising", "qubo"):
        _check(oracle, J, J, h, ptype, update, R, Rd, 4)


@pytest.mark.parametrize("update", ["sequential", "random"])
@pytest.mark.parametrize("kind,n", [
    ("ring", 40), ("ring", 516), ("lattice", 576), (12, 600), ("band", 160)])
@pytest.mark.parametrize("reads", [1300, 13000])
def test_many_items_agree_with_few(kind, n, reads, update):
    """The first reads of a batch of 5200 or 52000 chains and a batch of those
    reads alone: the same bits (the oracle has the latter above)."""
    from pysa_gb300 import Instance, PTBatch, pack_spins
    J, h = _problem(kind, n)
    betas = (1.0 / np.geomspace(0.3, 3.0, 4)).astype(np.float32)
    words = None
    got = []
    for rd in (reads, 9):
        b = PTBatch("qubo", [Instance(J, h, betas, rd)], sparse=True)
        if words is None:
            x = np.random.default_rng(1).integers(0, 2, (4 * rd, n), np.int8)
            words = pack_spins(x, "qubo", b.words)
        b.set_states(words[:4 * rd])
        b.run(3, seed=2, update=update)
        got.append(b.fetch())
    for k in got[1]:
        assert np.array_equal(got[0][k][:36], got[1][k]), k


@pytest.mark.parametrize("update", ["sequential", "random"])
def test_uneven_rows_match_oracle(oracle, update):
    """A few spins next to nearly all others, the rest next to few: grouped
    rows of 1 to 600 entries."""
    rng = np.random.default_rng(9)
    n = 700
    J = _graph(4, n, rng)
    for hub in (0, 1, 5, 350, 699):
        J[hub, rng.random(n) < rng.uniform(0.3, 0.9)] = rng.normal()
    J = np.triu(J, 1) + np.triu(J.T, 1)
    J = (J + J.T).astype(np.float32)
    h = rng.normal(size=n).astype(np.float32)
    _check(oracle, J, J, h, "ising", update, 3, 2, 4)


def test_rows_past_the_schedule_buffer():
    """Four neighbouring positions with more than 32 768 entries together:
    the schedule reads them from the rows, and the sweep equals the one that
    takes every quad by itself."""
    import scipy.sparse as sp
    from pysa_gb300 import Instance, PTBatch, pack_spins
    n, hubs = 12000, 4
    rng = np.random.default_rng(2)
    i = np.repeat(np.arange(hubs), n - hubs)
    j = np.tile(np.arange(hubs, n), hubs)
    k = np.arange(hubs, n - 1)
    A = sp.coo_matrix((np.r_[rng.integers(1, 4, len(i)), np.ones(len(k))],
                       (np.r_[i, k], np.r_[j, k + 1])), (n, n))
    A = sp.csr_matrix(A + A.T, dtype=np.float32)
    betas = (1.0 / np.geomspace(50.0, 3000.0, 3)).astype(np.float32)
    got = []
    for scheduled in (True, False):
        b = PTBatch("ising", [Instance(A, np.zeros(n, np.float32), betas,
                                       2)], sparse=True)
        if not scheduled:
            b.ws.perm = 0
        x = np.random.default_rng(3).integers(0, 2, (6, n), np.int8)
        b.set_states(pack_spins(x, "qubo", b.words))
        b.run(3, seed=4)
        got.append(b.fetch())
    for key in got[0]:
        assert np.array_equal(got[0][key], got[1][key]), key
    assert (got[0]["spins"] != pack_spins(x, "qubo", b.words)).any()
