"""Prepared fields and energies (k_fields) at the edges of its tiles, in every
tile variant, against the same sums in NumPy: f32 partial sums over 32 rows
accumulated in f64, rounded once."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _reference(ptype, J, h, x):
    s = 2.0 * x - 1.0 if ptype == "ising" else x.astype(np.float64)
    n = len(h)
    F = np.zeros((len(x), n))
    with np.errstate(invalid="ignore", over="ignore"):
        for j0 in range(0, n, 32):
            part = np.zeros((len(x), n), np.float32)
            for j in range(j0, min(j0 + 32, n)):
                live = s[:, j] != 0
                part[live] += s[live, j, None].astype(np.float32) * J.T[j]
            F += part
        H = (F + h).astype(np.float32)
        E = (s * (0.5 * F + h)).sum(1)  # every term, as the reference sums
    return H, E


def _run(ptype, problems, reads):
    from pysa_gb300 import Instance, PTBatch, pack_spins
    rng = np.random.default_rng(sum(reads))
    b = PTBatch(ptype, [Instance(J, h, np.ones(1, np.float32), r)
                        for (J, h), r in zip(problems, reads)],
                kernel="plain")
    xs = [rng.integers(0, 2, (r, len(h))).astype(np.uint8)
          for (_, h), r in zip(problems, reads)]
    b.set_states(np.concatenate([pack_spins(x, "qubo", b.words) for x in xs]))
    return (b.fields.cpu().numpy(), b.energies.cpu().numpy(), xs,
            b.chain_off)


# n and chains (reads of one replica): one lane, one word and one tile short,
# full and over; few chains (8-chain tiles, columns over a cluster), the
# 32-chain tile, and the 64-chain tiles of n <= 128 and n <= 32
@pytest.mark.parametrize("ptype,n,chains", [
    ("ising", 1, 1), ("qubo", 31, 7), ("ising", 33, 9), ("qubo", 255, 8),
    ("ising", 257, 17), ("ising", 1025, 5), ("qubo", 2300, 3),
    ("ising", 97, 9800), ("qubo", 260, 4900), ("ising", 513, 3300),
    ("qubo", 128, 19500), ("ising", 100, 19457), ("ising", 32, 19456),
    ("qubo", 5, 19470)])
@pytest.mark.parametrize("integer", [True, False])
def test_fields_match_numpy(ptype, n, chains, integer):
    rng = np.random.default_rng(n)
    J = rng.integers(-8, 9, (n, n)) if integer else rng.normal(size=(n, n))
    J = np.triu(J, 1).astype(np.float32)
    J = J + J.T
    h = (rng.integers(-9, 10, n) if integer else
         rng.normal(size=n)).astype(np.float32)
    H, E, (x,), _ = _run(ptype, [(J, h)], [chains])
    keep = np.arange(chains) if chains <= 64 else \
        np.r_[0:24, chains // 2:chains // 2 + 16, chains - 24:chains]
    Hr, Er = _reference(ptype, J, h, x[keep])
    if integer:
        assert (H[keep, :n] == Hr).all()
        assert (E[keep] == Er).all()
    else:
        # the accumulated pair is within 2^-47 of the f64 sum: at most the
        # other neighbour of a rounding tie
        assert (np.abs(H[keep, :n] - Hr) <= np.spacing(np.abs(Hr))).all()
        scale = (np.abs(J).sum() / 2 + np.abs(h).sum())
        assert (np.abs(E[keep] - Er) <=
                0.5 * np.spacing(np.abs(Er).astype(np.float32)) +
                2.0**-40 * scale).all()


def test_fields_of_uneven_instances_sharing_tiles():
    """Instances that begin inside a chain tile, of every size class."""
    rng = np.random.default_rng(5)
    sizes, reads = [3, 700, 64, 33, 1, 290], [1, 3, 40, 13, 2, 31]
    problems = []
    for n in sizes:
        J = np.triu(rng.integers(-8, 9, (n, n)), 1).astype(np.float32)
        problems.append((J + J.T, rng.integers(-9, 10, n).astype(np.float32)))
    H, E, xs, off = _run("ising", problems, reads)
    for (J, h), x, o in zip(problems, xs, off):
        Hr, Er = _reference("ising", J, h, x)
        assert (H[o:o + len(x), :len(h)] == Hr).all()
        assert (E[o:o + len(x)] == Er).all()


@pytest.mark.parametrize("ptype,chains", [("ising", 40), ("qubo", 40),
                                          ("qubo", 9800)])
def test_fields_with_infinite_and_huge_couplings(ptype, chains):
    """A zero spin leaves an infinite coupling out of the fields (an energy
    has a term for every spin: 0 times infinity is NaN); sums past f32 keep
    the f64 accumulation."""
    n = 70
    rng = np.random.default_rng(1)
    J = np.triu(rng.integers(-8, 9, (n, n)), 1).astype(np.float32)
    J[3, 40] = np.inf
    J[50:60, 65] = 3e38
    J = np.triu(J, 1) + np.triu(J, 1).T
    h = np.zeros(n, np.float32)
    h[20] = -np.inf
    H, E, (x,), _ = _run(ptype, [(J, h)], [chains])
    keep = np.arange(min(chains, 64))
    Hr, Er = _reference(ptype, J, h, x[keep])
    np.testing.assert_array_equal(H[keep, :n], Hr)
    with np.errstate(over="ignore"):
        np.testing.assert_array_equal(E[keep], Er.astype(np.float32))
