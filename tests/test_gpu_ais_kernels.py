"""Annealed importance sampling in every kernel form (a thread, a warp, or a
shared warp per sample) at the edges of their sizes, against the oracle; the
couplings are half-integers, so every field is exact and samples must agree
bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# n: one spin, each padded width of the thread-per-sample kernel +- 1, each
# column count of the warp-per-sample kernel +- 1, the widest it takes and
# past it; sample counts either side of a warp, a CTA and the switch between
# the forms (4096 for n <= 32)
@pytest.mark.parametrize("update", ["sequential", "random"])
@pytest.mark.parametrize("ref", ["uniform", "bernoulli"])
@pytest.mark.parametrize("ptype,n,ns", [
    ("ising", 1, 3), ("qubo", 5, 33), ("ising", 32, 40), ("qubo", 33, 9),
    ("ising", 64, 5), ("qubo", 65, 6), ("ising", 128, 7), ("qubo", 129, 17),
    ("ising", 220, 3), ("qubo", 221, 3),
    ("ising", 1, 4200), ("qubo", 8, 4097), ("ising", 9, 4225),
    ("qubo", 16, 4100), ("ising", 23, 4100), ("qubo", 25, 4200)])
def test_ais_forms_match_oracle(oracle, ptype, n, ns, ref, update):
    from pysa_gb300.engine import run_ais
    rng = np.random.default_rng(n + ns)
    J = np.triu(rng.integers(-2, 3, (n, n)), 1).astype(np.float32)
    J = 0.5 * (J + J.T)
    h = 0.5 * rng.integers(-2, 3, n).astype(np.float32)
    x0 = rng.integers(0, 2, (ns, n)).astype(np.float32)
    x0 = 2 * x0 - 1 if ptype == "ising" else x0
    # zero, tiny and ordinary inverse temperatures
    temps = np.array([0.0, 1e-35, 0.02, 0.3, 0.7, 1.0], np.float32)
    kw = dict(seed=77, update=update, p=0.3,
              order="standard" if n % 2 else "reference")
    s, lw = run_ais(ptype, J, h, temps, x0, reference=ref, **kw)
    ws, wlw = oracle.ais_run(ptype, J, h, temps, x0, ref=ref, **kw)
    assert np.array_equal(s, ws)
    np.testing.assert_allclose(lw, wlw, rtol=1e-9, atol=1e-9)


def test_ais_infinite_field_and_negative_temperature(oracle):
    """A pinned spin (infinite field) and a step of negative inverse
    temperature, which the thresholds leave to the exact rule."""
    from pysa_gb300.engine import run_ais
    rng = np.random.default_rng(2)
    n = 20
    J = np.triu(rng.integers(-2, 3, (n, n)), 1).astype(np.float32)
    J = J + J.T
    h = np.zeros(n, np.float32)
    h[4] = np.inf
    temps = np.array([-0.2, 0.4, 1.0], np.float32)
    for ns in (50, 4200):
        x0 = 2.0 * rng.integers(0, 2, (ns, n)).astype(np.float32) - 1
        with np.errstate(invalid="ignore"):
            s, _ = run_ais("ising", J, h, temps, x0, seed=5)
            ws, _ = oracle.ais_run("ising", J, h, temps, x0, seed=5)
        assert np.array_equal(s, ws)
