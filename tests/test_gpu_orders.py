"""Visiting orders made in rounds of independent swaps equal the sequential
Fisher-Yates of the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# the first orders past the resident sweep, a thread's second swap (512 and
# 1024 threads), and either side of the widest order held in shared memory
@pytest.mark.parametrize("n", [65, 511, 512, 513, 1025, 2048, 2049, 4097,
                               29056, 29057])
def test_orders_match_oracle(oracle, n):
    from pysa_gb300 import Instance, PTBatch
    # no couplings: the order depends on the seed, the instance and n alone
    insts = [Instance(np.broadcast_to(np.float32(0.0), (k, k)),
                      np.zeros(k, np.float32), np.ones(1, np.float32), 1)
             for k in ((3, n) if n < 8192 else (n,))]
    b = PTBatch("ising", insts, kernel="plain", perm_slots=2)
    b.set_states(np.zeros((len(insts), b.words), np.uint32))
    b.run(2, seed=5, update="random", use_pt=False)
    b.check_status()
    perm = b.perm.cpu().numpy().reshape(2, len(insts), b.max_n)
    for sweep in range(2):
        for i, x in enumerate(insts):
            k = len(x.h)
            want = oracle.permutation(5, i, sweep, k)
            assert (perm[sweep, i, :k] == want).all()
