"""Leaf hashes of matrix rows: widths around the 136-byte block (a row that ends
before, on and after a block's end, odd and even word counts), and row counts that
fill a warp's 32 rows, miss them and leave a ragged last warp.  Roots against the
oracle (a root binds every leaf)."""
import numpy as np
import pytest

from oracle import oracle as O
from basefold_gpu import rand

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w", [2, 8, 9, 16, 17, 18, 25, 26, 34, 51])
def test_binary_rows(built_lib, w):
    bg = built_lib
    for n, log2_c in [(0, 0), (3, 1), (4, 1), (6, 0), (5, 2)]:
        data = rand.random_elems(w << n, 7000 + 10 * w + n)
        pcs = bg.Basefold.setup(bg.BasefoldConfig(bg.BinaryReedSolomonCode(128, log2_c, n)))
        assert pcs.commit(data, width=w).root == O.commit_root(n, log2_c, data, width=w), (n, log2_c)


@pytest.mark.parametrize("w", [2, 3, 31, 32, 33, 34, 35, 66, 67, 68, 69, 70, 102, 103])
def test_prime_rows(built_lib, w):
    from basefold_gpu import BasefoldConfig, prime

    for n, log2_c in [(1, 0), (3, 1), (4, 1), (6, 0), (5, 2)]:
        data = np.random.default_rng(100 * w + n).integers(0, O.BB_P, size=(1 << n, w), dtype=np.uint64).astype(np.uint32)
        point = np.zeros((n, 5), np.uint32)
        pcs = prime.BabyBearBasefold.setup(BasefoldConfig(prime.ReedSolomonCode(128, log2_c, n)), device=0)
        assert pcs.commit(data).root == O.bb_harness_prepare(n, log2_c, data, point)[0], (n, log2_c)
