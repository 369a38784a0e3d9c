"""The resident sweep of small instances (n <= 64, all sweeps of a read in
one launch) and log-omega inside the fused launches, against the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _problem(rng, n, integer):
    J = rng.integers(-4, 5, (n, n)) if integer else rng.normal(size=(n, n))
    J = np.triu(J, 1).astype(np.float32)
    h = (rng.integers(-4, 5, n) if integer else
         rng.normal(size=n)).astype(np.float32)
    return J + J.T, h


def _start(oracle, rng, ptype, J, h, Rd, R):
    x = rng.integers(0, 2, (Rd, R, len(h))).astype(np.float32)
    x = 2 * x - 1 if ptype == "ising" else x
    e = np.array([[oracle.energy64(J, h, s) for s in r] for r in x],
                 np.float32)
    return x, e


def _compare(oracle, ptype, problems, shapes, update, sweeps, betas_of,
             log_omega=False, use_pt=True, kernel="auto", split=None,
             exchange_every=1):
    from pysa_gb300 import Instance, PTBatch, pack_spins, unpack_spins
    rng = np.random.default_rng(sum(R * Rd for R, Rd in shapes))
    insts, xs, es = [], [], []
    for (J, h), (R, Rd) in zip(problems, shapes):
        insts.append(Instance(J, h, betas_of(R), Rd))
        x, e = _start(oracle, rng, ptype, J, h, Rd, R)
        xs.append(x)
        es.append(e)
    b = PTBatch(ptype, insts, kernel=kernel)
    b.set_states(np.concatenate([
        pack_spins(x, ptype, b.words).reshape(-1, b.words) for x in xs]),
        np.concatenate([e.reshape(-1) for e in es]))
    for k in (split or [sweeps]):
        b.run(k, seed=99, update=update, use_pt=use_pt, log_omega=log_omega,
              exchange_every=exchange_every)
    got = b.fetch()
    read0 = 0
    for i, ((J, h), (R, Rd)) in enumerate(zip(problems, shapes)):
        c0, n = int(b.chain_off[i]), len(h)
        w = oracle.pt_run(ptype, J, h, betas_of(R), xs[i], es[i],
                          np.tile(np.arange(R, dtype=np.int32), (Rd, 1)),
                          seed=99, num_sweeps=sweeps, update=update,
                          use_pt=use_pt, log_omega=log_omega, inst=i,
                          exchange_every=exchange_every)
        s = slice(c0, c0 + R * Rd)
        sp = unpack_spins(got["spins"][s], n, ptype, np.float32)
        assert (sp.reshape(Rd, R, n) == w["spins"]).all(), i
        assert (got["energies"][s].reshape(Rd, R) == w["energies"]).all(), i
        assert (got["beta_idx"][s].reshape(Rd, R) == w["beta_idx"]).all(), i
        assert (got["best_energy"][s].reshape(Rd, R) ==
                w["best_energy"]).all(), i
        assert (got["best_sweep"][s].reshape(Rd, R) ==
                w["best_sweep"]).all(), i
        bsp = unpack_spins(got["best_spins"][s], n, ptype, np.float32)
        assert (bsp.reshape(Rd, R, n) == w["best_spins"]).all(), i
        if log_omega:
            # sums of at most R f32 terms in f64, in another order
            lw = got["log_omega"][read0:read0 + Rd]
            scale = np.abs(w["energies"]).max() * np.abs(betas_of(R)).max()
            np.testing.assert_allclose(lw, w["log_omega"], rtol=0,
                                       atol=R * R * scale * 2.0**-50)
        read0 += Rd
    return b


def _geometric(R):
    b = (1.0 / np.geomspace(0.3, 3.0, R)).astype(np.float32)
    if R > 2:
        b[-1] = 0.0
    return b


# one position, half and both halves of the lanes, each +- 1; one chain, one
# per warp, and more chains than the CTA's 31 chain warps
@pytest.mark.parametrize("update", ["sequential", "random"])
@pytest.mark.parametrize("ptype,n,R,Rd", [
    ("ising", 1, 1, 1), ("qubo", 2, 3, 2), ("ising", 31, 4, 3),
    ("qubo", 32, 5, 2), ("ising", 33, 31, 2), ("qubo", 47, 32, 2),
    ("ising", 63, 33, 1), ("qubo", 64, 70, 2)])
def test_small_matches_oracle(oracle, ptype, n, R, Rd, update):
    J, h = _problem(np.random.default_rng(n), n, True)
    _compare(oracle, ptype, [(J, h)], [(R, Rd)], update, 13, _geometric,
             kernel="plain", log_omega=True)


def test_small_float_couplings(oracle):
    """Real couplings: the same f32 field updates and energy sums as the
    oracle's local-field form, so only rounding-free decisions differ."""
    from pysa_gb300 import Instance, PTBatch, pack_spins
    rng = np.random.default_rng(8)
    J, h = _problem(rng, 40, False)
    x, e = _start(oracle, rng, "ising", J, h, 4, 8)
    out = []
    for phases in (0, None):
        b = PTBatch("ising", [Instance(J, h, _geometric(8), 4)],
                    kernel="plain")
        b.set_states(pack_spins(x, "ising", b.words), e.reshape(-1))
        if phases is None:  # sweep and exchange apart: the plain kernel
            from pysa_gb300 import _lib
            for _ in range(30):
                for ph in (1, 2):
                    o = _lib.Options(5, _lib.RANDOM, 1, 0, 0, ph, 0, 1)
                    _lib.check(b.lib.pysa_gb_sweeps(
                        _lib.ref(b.p), _lib.ref(b.s), _lib.ref(b.ws),
                        _lib.ref(o), 1, b._stream.cuda_stream), "sweeps")
        else:
            b.run(30, seed=5, update="random")
        out.append((b.fetch(), b.fields[:, :40].cpu().numpy()))
    for k in out[0][0]:
        assert (out[0][0][k] == out[1][0][k]).all(), k
    assert (out[0][1] == out[1][1]).all()


def test_small_beside_tensor_cores_and_uneven_replicas(oracle):
    """One batch of tensor-core and small instances, the small ones with
    more replicas than the batch's average read; split over three calls."""
    rng = np.random.default_rng(2)
    problems = [_problem(rng, n, True) for n in (20, 130, 64, 63, 5)]
    shapes = [(8, 2), (4, 6), (8, 3), (40, 1), (3, 5)]
    for update in ("sequential", "random"):
        b = _compare(oracle, "qubo", problems, shapes, update, 9, _geometric,
                     split=[4, 1, 4])
        assert b.tc


@pytest.mark.parametrize("kw", [dict(use_pt=False), dict(exchange_every=3)])
def test_small_exchange_options(oracle, kw):
    J, h = _problem(np.random.default_rng(3), 30, True)
    _compare(oracle, "ising", [(J, h)], [(6, 3)], "random", 11, _geometric,
             **kw)


@pytest.mark.parametrize("update", ["sequential", "random"])
@pytest.mark.parametrize("n,R,use_pt", [(100, 32, True), (600, 16, True),
                                        (130, 8, False)])
def test_log_omega_inside_the_tensor_core_launch(oracle, n, R, use_pt,
                                                 update):
    J, h = _problem(np.random.default_rng(n), n, True)
    _compare(oracle, "qubo", [(J, h)], [(R, 5)], update, 6, _geometric,
             log_omega=True, use_pt=use_pt)
