"""Energies of long AIS runs are carried in 64 bits in every kernel form."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("update", ["sequential", "random"])
@pytest.mark.parametrize("n,samples", [
    (12, 64), (40, 64),  # a warp per sample
    (12, 6000),          # a thread per sample
    (40, 30000)])        # several samples per warp
def test_energy_sums_keep_53_bits(n, samples, update):
    """Opposite fields of 2^40, 2^28 and 2^14 on pairs of uncoupled spins, and
    multiples of 2^-10 elsewhere: every energy is a multiple of 2^-10 below
    2^42, exact in 64 bits but not in 48.  Where all pairs are aligned at the
    end the energy is small and has to be exact, whatever the sums on the way
    passed through."""
    from pysa_gb300 import Instance, PTBatch, _lib, pack_spins, unpack_spins
    import torch
    rng = np.random.default_rng(n + samples)
    h = rng.integers(-2000, 2001, n) * 2.0**-10
    h[:6] = [2.0**40, -2.0**40, 2.0**28, -2.0**28, 2.0**14, -2.0**14]
    J = np.zeros((n, n))
    J[6:, 6:] = np.triu(rng.integers(-500, 501, (n - 6, n - 6)) * 2.0**-10, 1)
    J = J + J.T
    x = 2 * rng.integers(0, 2, (samples, n)) - 1
    x[:, 1:6:2] = x[:, 0:6:2]  # aligned: the first energies are small
    temps = (2.0**-44 * np.arange(1, 61) / 60).astype(np.float32)
    b = PTBatch("ising", [Instance(J.astype(np.float32), h.astype(np.float32),
                                   np.ones(1, np.float32), samples)],
                perm_slots=len(temps), kernel="plain")
    e0 = ((x @ J) / 2 * x + x * h).sum(axis=1)
    b.set_states(pack_spins(x, "ising", b.words), e0.astype(np.float32))
    t = torch.from_numpy(temps).to(b.device)
    lw = torch.zeros(samples, dtype=torch.float64, device=b.device)
    opts = _lib.AisOptions(5, _lib.RANDOM if update == "random" else
                           _lib.SEQUENTIAL, 0, 0, len(temps), 0.5, samples, 0)
    _lib.check(b.lib.pysa_gb_ais(_lib.ref(b.p), _lib.ref(b.s), _lib.ref(b.ws),
                                 _lib.ref(opts), t.data_ptr(), lw.data_ptr(),
                                 b._stream.cuda_stream), "ais")
    got = b.fetch()
    s = unpack_spins(got["spins"], n, "ising", np.float64)
    small = (s[:, 0:6:2] == s[:, 1:6:2]).all(axis=1)
    assert small.sum() > 2 and not np.array_equal(s, x)
    want = ((s @ J) / 2 * s + s * h).sum(axis=1)  # exact in 64 bits
    assert np.array_equal(got["energies"][small], want[small])
