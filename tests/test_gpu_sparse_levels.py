"""The sparse-row sweep's level schedule: quads of visiting positions run in
parallel only where no flip of one is read by another, so every graph shape
keeps the oracle's trajectory bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _graph(kind, n, rng):
    J = np.zeros((n, n), np.float32)
    if kind == "ring":      # every quad depends on the one before
        i = np.arange(n)
        if n > 1:
            J[i, (i + 1) % n] = 1.0
    elif kind == "star":    # spin 0 next to every other: rows past 32 entries
        J[0, 1:] = rng.integers(1, 4, n - 1)
    elif kind == "empty":
        pass
    elif kind == "clusters":  # full blocks of 7: in-quad and in-level words
        for b in range(0, n, 7):
            J[b:b + 7, b:b + 7] = rng.normal(size=J[b:b + 7, b:b + 7].shape)
    else:                   # random rows of up to `kind` entries
        for r in range(n):
            c = rng.choice(n, min(kind // 2, n), replace=False)
            J[r, c] = rng.normal(size=len(c))
    J = np.triu(J, 1)
    return (J + J.T).astype(np.float32)


def _check(oracle, J, Jo, h, ptype, update, R, Rd, sweeps, null_perm=False,
           perm_slots=1):
    from pysa_gb300 import Instance, PTBatch, pack_spins, unpack_spins
    n = len(h)
    rng = np.random.default_rng(n + R)
    betas = (1.0 / np.geomspace(0.3, 3.0, R)).astype(np.float32)
    if R > 2:
        betas[-1] = 0.0
    x0 = rng.integers(0, 2, (Rd, R, n)).astype(np.float32)
    x0 = 2 * x0 - 1 if ptype == "ising" else x0
    e0 = np.array([[oracle.energy64(Jo, h, s) for s in r] for r in x0],
                  np.float32)
    b = PTBatch(ptype, [Instance(J, h, betas, Rd)], sparse=True,
                perm_slots=perm_slots)
    if null_perm:
        b.ws.perm = 0
    b.set_states(pack_spins(x0, ptype, b.words), e0.reshape(-1))
    b.run(sweeps, seed=n, update=update)
    got = b.fetch()
    want = oracle.pt_run(ptype, Jo, h, betas, x0, e0,
                         np.tile(np.arange(R, dtype=np.int32), (Rd, 1)),
                         seed=n, num_sweeps=sweeps, update=update)
    sp = unpack_spins(got["spins"].reshape(Rd, R, -1), n, ptype, np.float32)
    assert (sp == want["spins"]).all()
    assert (got["energies"].reshape(Rd, R) == want["energies"]).all()
    assert (got["beta_idx"].reshape(Rd, R) == want["beta_idx"]).all()
    assert (got["best_energy"].reshape(Rd, R) == want["best_energy"]).all()


# 1 .. 9 spins: no schedule, the first schedules; word and quad edges; one,
# two and four warps' worth of quads; 31, 32 and 33 chains of an item
@pytest.mark.parametrize("update", ["sequential", "random"])
@pytest.mark.parametrize("kind,n,R,Rd", [
    ("ring", 1, 2, 1), ("ring", 5, 3, 2), ("ring", 7, 1, 1),
    ("ring", 8, 4, 2), ("clusters", 9, 3, 1), ("ring", 33, 31, 1),
    ("star", 40, 32, 1), ("star", 300, 11, 3), ("empty", 130, 3, 2),
    ("clusters", 515, 5, 2), (8, 513, 4, 2), (14, 600, 3, 1),
    (30, 700, 3, 1), (6, 2050, 2, 1)])
def test_levels_match_oracle(oracle, kind, n, R, Rd, update):
    rng = np.random.default_rng(n)
    J = _graph(kind, n, rng)
    h = rng.normal(size=n).astype(np.float32)
    _check(oracle, J, J, h, "qubo" if n % 2 else "ising", update, R, Rd, 4)


@pytest.mark.parametrize("update", ["sequential", "random"])
def test_one_sided_entries_keep_their_order(oracle, update):
    """Entries without their mirror image (couplings symmetric only to a
    tolerance): a spin read by an earlier position is flipped after it."""
    rng = np.random.default_rng(3)
    n = 260
    J = _graph(6, n, rng)
    J[rng.random((n, n)) < 0.5] = 0.0   # row i of J^T is what spin i reads
    h = rng.normal(size=n).astype(np.float32)
    _check(oracle, J, np.ascontiguousarray(J.T), h, "ising", update, 4, 2, 5,
           perm_slots=3)


def test_sequential_without_order_workspace(oracle):
    rng = np.random.default_rng(4)
    J = _graph(6, 90, rng)
    h = rng.normal(size=90).astype(np.float32)
    _check(oracle, J, J, h, "ising", "sequential", 4, 2, 4, null_perm=True)
