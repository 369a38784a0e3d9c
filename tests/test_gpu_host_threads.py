"""Two host threads sweep batches of different sizes at the same time, each
on a stream of its own: neither's launches fail for the other's shared-memory
needs, and the results are those of each batch alone."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _ring(n):
    import scipy.sparse as sp
    i = np.arange(n)
    A = sp.coo_matrix((np.ones(n, np.float32), (i, (i + 1) % n)), (n, n))
    return sp.csr_matrix(A + A.T)


def _dense(n):
    J = np.triu(np.random.default_rng(n).integers(-4, 5, (n, n)), 1)
    return (J + J.T).astype(np.float32)


def _batch(kind, n, R, reads):
    from pysa_gb300 import Instance, PTBatch
    betas = (1.0 / np.geomspace(0.5, 8.0, R)).astype(np.float32)
    J = _ring(n) if kind == "sparse" else _dense(n)
    return PTBatch("ising", [Instance(J, np.zeros(n, np.float32), betas,
                                      reads)], sparse=kind == "sparse")


def _steps(kind, shape, count, errors, gate, out):
    """count sweeps (or annealing runs) one call each, from a fixed state."""
    import torch
    from pysa_gb300 import _lib
    try:
        with torch.cuda.stream(torch.cuda.Stream()):
            b = _batch(kind, *shape)
            words = np.zeros((b.num_chains, b.words), np.uint32)
            b.set_states(words)
            st = b._stream.cuda_stream
            temps = torch.ones(1, device=b.device)
            lw = torch.zeros(b.num_chains, dtype=torch.float64,
                             device=b.device)
            opts = _lib.Options(3, _lib.SEQUENTIAL, 1, 0, 0, 0, 0, 1)
            ais = _lib.AisOptions(3, _lib.SEQUENTIAL, 0, 0, 1, 0.5, shape[2],
                                  0)
            torch.cuda.synchronize()
            gate.wait()
            for _ in range(count):
                if kind == "ais":
                    _lib.check(b.lib.pysa_gb_ais(
                        _lib.ref(b.p), _lib.ref(b.s), _lib.ref(b.ws),
                        _lib.ref(ais), temps.data_ptr(), lw.data_ptr(), st),
                        "ais")
                else:
                    _lib.check(b.lib.pysa_gb_sweeps(
                        _lib.ref(b.p), _lib.ref(b.s), _lib.ref(b.ws),
                        _lib.ref(opts), 1, st), "sweeps")
            out.append(b.fetch())
    except Exception as e:  # noqa: BLE001 (reported by the test)
        errors.append(e)


@pytest.mark.parametrize("kind,large,small,count", [
    ("small", (40, 256, 1), (24, 2, 1), 3000),
    ("ais", (200, 1, 16), (140, 1, 16), 3000),
    ("sparse", (12900, 2, 1), (64, 2, 1), 600)])
def test_two_threads_of_different_sizes(kind, large, small, count):
    errors, alone = [], []
    for shape in (large, small):
        _steps(kind, shape, count, errors, threading.Barrier(1), alone)
    assert not errors, errors
    gate = threading.Barrier(2)
    outs = [[], []]
    ts = [threading.Thread(target=_steps, args=(kind, s, count, errors, gate,
                                                o))
          for s, o in zip((large, small), outs)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not errors, errors
    both = [o[0] for o in outs]
    for a, b in zip(alone, both):
        for k in a:
            assert np.array_equal(a[k], b[k]), k


def test_two_threads_fetch_one_batch():
    """Results of over 4 MB pass a pinned buffer: two threads that read one
    batch at the same time each get its state, not the other's pieces."""
    from pysa_gb300 import Instance, PTBatch, pack_spins
    n, R, reads = 512, 8, 16384
    b = PTBatch("ising", [Instance(_dense(n), np.zeros(n, np.float32),
                                   np.geomspace(0.01, 1.0, R).astype(
                                       np.float32), reads)], kernel="plain")
    x = np.random.default_rng(0).integers(0, 2, (R * reads, n), np.int8)
    words = pack_spins(x, "qubo", b.words)
    b.set_states(words)
    b.run(2, seed=1)
    want = b.fetch()
    assert not np.array_equal(want["spins"], want["best_spins"])
    wrong, errors = [], []

    def read():
        try:
            for _ in range(40):
                got = b.fetch()
                wrong.append(not all(np.array_equal(got[k], want[k])
                                     for k in want))
        except Exception as e:  # noqa: BLE001 (reported by the test)
            errors.append(e)

    ts = [threading.Thread(target=read) for _ in range(2)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not errors, errors
    assert len(wrong) == 80 and not any(wrong)
