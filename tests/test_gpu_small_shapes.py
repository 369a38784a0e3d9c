"""Small dense instances in every form their sweep takes, against the oracle:
rows of 32 and 64 columns, one warp a read, a CTA's chains in several turns,
clusters, reads of far more replicas than the batch's average, and the sweep in
separate launches that many reads in short calls take."""
import numpy as np
import pytest

from test_gpu_small import _compare, _geometric, _problem

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("update", ["sequential", "random"])
@pytest.mark.parametrize("n,shapes,sweeps", [
    (32, [(1, 5)], 20),                       # no helper warp in order
    (33, [(1, 5)], 20),
    (8, [(16, 700)], 16),                     # several CTAs an SM, turns
    (40, [(32, 400)], 16),
    (31, [(512, 2)], 16),                     # a cluster, a read in turns
    (24, [(1, 300), (64, 2)], 16),            # R above cap: its own launch
    (64, [(3, 40), (200, 1), (1, 10)], 16),
    (24, [(1, 6000)], 1),                     # short call: launches per sweep
    (9, [(2, 30), (500, 1)], 3)])
def test_shapes_match_oracle(oracle, n, shapes, sweeps, update):
    rng = np.random.default_rng(n + len(shapes))
    problems = [_problem(rng, n, True) for _ in shapes]
    _compare(oracle, "ising", problems, shapes, update, sweeps, _geometric,
             kernel="plain")


def test_other_instances_left_alone(oracle):
    """Small instances of mixed replica counts beside tensor-core ones."""
    rng = np.random.default_rng(3)
    problems = [_problem(rng, n, True) for n in (20, 100, 50)]
    _compare(oracle, "qubo", problems, [(2, 40), (4, 8), (120, 1)],
             "sequential", 16, _geometric)


@pytest.mark.parametrize("update", ["sequential", "random"])
@pytest.mark.parametrize("n,R,reads", [(24, 1, 6000), (60, 4, 3000)])
def test_resident_and_launched_sweeps_agree(n, R, reads, update):
    """Real couplings: eight calls of one sweep (three launches each) and one
    of eight (resident) give the same bits."""
    from pysa_gb300 import Instance, PTBatch, pack_spins
    rng = np.random.default_rng(n)
    J, h = _problem(rng, n, False)
    b = PTBatch("ising", [Instance(J, h, _geometric(R), reads)],
                kernel="plain")
    words = pack_spins(rng.integers(0, 2, (R * reads, n)), "qubo", b.words)
    got = []
    for calls in ([1] * 8, [8]):
        b.set_states(words)
        for k in calls:
            b.run(k, seed=4, update=update)
        got.append(b.fetch())
    for k in got[0]:
        assert np.array_equal(got[0][k], got[1][k]), k
