"""Real couplings on the tensor-core sweep: a run's outputs are the same bit
for bit however its work is spread over CTAs and launches.

At fold 2 (512 < n <= 1024) the two forms in which a 64-spin block may be
decided round a field's corrections differently, so there the form of every
block has to follow from its own item alone, not from what the CTA swept
before.  At folds 1 and 4 the forms round alike, and forcing one changes
nothing."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture
def lib():
    from pysa_gb300 import _lib
    lib = _lib.load()
    yield lib
    _lib.check(lib.pysa_gb_set_tc_max_ctas(0), "max ctas reset")
    _lib.check(lib.pysa_gb_set_decision_mode(0), "mode reset")


def _batch(sizes, R, reads):
    from pysa_gb300 import Instance, PTBatch, pack_spins
    rng = np.random.default_rng(sum(sizes))
    insts, words = [], []
    betas = (1.0 / np.geomspace(1.0, 3.5, R)).astype(np.float32)
    for n in sizes:
        J = np.triu(rng.normal(size=(n, n)) / np.sqrt(n), 1)
        J = (J + J.T).astype(np.float32)
        insts.append(Instance(J, np.zeros(n, np.float32), betas, reads))
    b = PTBatch("ising", insts, kernel="tc")
    assert b.tc_terms == 2 and b.ws.tc_fusable == 1
    for n in sizes:
        words.append(pack_spins(rng.integers(0, 2, (R * reads, n)), "qubo",
                                b.words))
    return b, np.concatenate(words)


def _run(b, words, sweeps, update):
    b.set_states(words)
    b.run(sweeps, seed=3, update=update)
    return b.fetch()


@pytest.mark.parametrize("update", ["sequential", "random"])
@pytest.mark.parametrize("sizes", [
    (516, 705, 969),             # fold 2, last blocks of 4, 1 and 9 spins
    (516, 139, 705, 1158, 969),  # every fold
    (705,)])                     # one size: wrap-around units
def test_spread_of_the_work_changes_nothing(lib, sizes, update):
    from pysa_gb300 import _lib
    b, words = _batch(sizes, 8, 256 if len(sizes) == 1 else 64)
    want = None
    for ctas, unit in ((0, 0), (2, 0), (7, 0), (0, 0), (19, 0), (5, 3),
                       (0, 20)):
        _lib.check(lib.pysa_gb_set_tc_max_ctas(ctas), "max ctas")
        b.ws.tc_unit_sweeps = unit
        got = _run(b, words, 20, update)
        want = want or got
        for k in want:
            assert np.array_equal(got[k], want[k]), (k, ctas, unit)


@pytest.mark.parametrize("update", ["sequential", "random"])
@pytest.mark.parametrize("n", [139, 328, 512, 1045, 1158])
def test_forms_agree_at_folds_1_and_4(lib, n, update):
    from pysa_gb300 import _lib
    b, words = _batch((n,), 8, 16)
    want = None
    for mode in (0, 1, 2):
        _lib.check(lib.pysa_gb_set_decision_mode(mode), "mode")
        got = _run(b, words, 12, update)
        want = want or got
        for k in want:
            assert np.array_equal(got[k], want[k]), (k, mode)
