"""Initial states drawn in one call take the same numbers of NumPy's global
stream as one call a sample, and leave it at the same place."""
import numpy as np
import pytest

from pysa_gb300 import ais


@pytest.mark.parametrize("ptype", ["ising", "qubo"])
@pytest.mark.parametrize("n,count", [(1, 1), (7, 3), (96, 50), (33, 0)])
def test_one_call_equals_one_a_sample(ptype, n, count):
    for many, one in (
            (lambda: ais.uniform_samples(n, ptype, count),
             lambda: ais.uniform_prob_initialization(n, ptype)),
            (lambda: ais.bernoulli_samples(n, ptype, count, (0.3,)),
             lambda: ais.bernoulli_prob_initialization(n, ptype, (0.3,)))):
        np.random.seed(5)
        want = [one() for _ in range(count)]
        end = np.random.randint(1 << 30)
        np.random.seed(5)
        got = many()
        assert got.shape == (count, n)
        assert all(np.array_equal(g, w) for g, w in zip(got, want))
        assert np.random.randint(1 << 30) == end


def test_reads_in_one_call():
    for R, N, reads in ((4, 24, 1), (3, 17, 9)):
        np.random.seed(1)
        want = np.stack([np.random.randint(2, size=(R, N))
                         for _ in range(reads)])
        np.random.seed(1)
        assert np.array_equal(np.random.randint(2, size=(reads, R, N)), want)


def test_unknown_problem_type_is_refused():
    for f in (ais.uniform_samples, ais.bernoulli_samples):
        with pytest.raises(ValueError):
            f(4, "potts", 2)
