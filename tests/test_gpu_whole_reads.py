"""Tensor-core work items of whole reads when the replicas do not divide the
chains per CTA: some chain slots stay empty, the exchange and log-omega run
inside the launch, and the trajectory is the oracle's."""
import numpy as np
import pytest

from test_gpu_small import _compare, _geometric, _problem

pytestmark = pytest.mark.gpu


# every fold (128, 64 and 32 chains per CTA): reads that leave few slots, the
# most that still leaves one read, one read short of and past a full item,
# and replicas past a CTA's chains (the exchange stays outside)
@pytest.mark.parametrize("update", ["sequential", "random"])
@pytest.mark.parametrize("n,R,Rd,fused", [
    (70, 9, 14, True), (70, 9, 15, True), (64, 127, 2, True),
    (200, 40, 3, True), (200, 129, 1, False), (600, 24, 5, True),
    (1030, 24, 2, True), (1030, 33, 1, False)])
def test_whole_reads_match_oracle(oracle, n, R, Rd, fused, update):
    J, h = _problem(np.random.default_rng(n), n, True)
    b = _compare(oracle, "qubo", [(J, h)], [(R, Rd)], update,
                 4 if n < 1000 else 2, _geometric, log_omega=True)
    assert b.tc and bool(b.ws.tc_fusable) == fused


def test_whole_reads_of_uneven_instances(oracle):
    rng = np.random.default_rng(1)
    problems = [_problem(rng, n, True) for n in (65, 513, 130)]
    b = _compare(oracle, "ising", problems, [(7, 3), (12, 2), (30, 5)],
                 "sequential", 5, _geometric, split=[2, 3])
    assert b.ws.tc_fusable


def test_few_slots_used_by_many_reads_stays_unfused():
    """Half the chain slots empty over several waves costs more than a launch
    per sweep."""
    from pysa_gb300 import Instance, PTBatch
    J, h = _problem(np.random.default_rng(0), 512, True)
    b = PTBatch("ising", [Instance(J, h, _geometric(72), 400)])
    assert b.tc and not b.ws.tc_fusable
    b = PTBatch("ising", [Instance(J, h, _geometric(72), 100)])
    assert b.ws.tc_fusable
