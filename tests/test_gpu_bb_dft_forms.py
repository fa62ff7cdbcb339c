"""The wide BabyBear DFT's first pass, which loads data rows with the copies that its
first layers would make: blowups from none to more layers than a tile has, and
passes of few and many layers.  Roots against the oracle (a root binds the codeword)."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,log2_c,w", [(0, 1, 17), (0, 9, 18), (1, 8, 20), (2, 0, 33), (3, 5, 64), (8, 2, 17), (9, 3, 20),
                                        (12, 1, 40), (13, 0, 32), (11, 4, 31)])
def test_wide_encodes_match_the_oracle(built_lib, n, log2_c, w):
    from basefold_gpu import BasefoldConfig, prime

    data = np.random.default_rng(50 * n + w).integers(0, O.BB_P, size=(1 << n, w), dtype=np.uint64).astype(np.uint32)
    data[0, :3] = (0, 1, O.BB_P - 1)
    data[-1] = O.BB_P - 1
    point = np.zeros((n, 5), np.uint32)
    pcs = prime.BabyBearBasefold.setup(BasefoldConfig(prime.ReedSolomonCode(128, log2_c, n)), device=0)
    assert pcs.commit(data).root == O.bb_harness_prepare(n, log2_c, data, point)[0]
