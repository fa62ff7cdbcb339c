"""Merkle trees and open tails at the sizes where the hashing form changes: one
warp per hash (up to 8 in a block), a pair of lanes (up to 64), one thread
(above); one block (up to 2^7 nodes), a cluster of eight (2^8 .. 2^12), subtree
launches of 2^6 .. 2^9 leaves per block above.  Whole proofs against the
oracle's bytes."""
import numpy as np
import pytest

from oracle import oracle as O
from basefold_gpu import rand

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,log2_c", [(n, 1) for n in range(0, 14)] + [(2, 0), (7, 0), (10, 0), (4, 3), (8, 3), (11, 4),
                                                                      (15, 2), (17, 1)])
def test_tree_and_tail_forms_give_the_oracle_proof(built_lib, n, log2_c):
    bg = built_lib
    data = rand.random_elems((1 << n) + n, 9100 + 16 * n + log2_c)
    evals, point = data[: 1 << n], data[1 << n:]
    root_o, values_o, blob = O.harness_prepare(n, log2_c, evals, point)
    want = O.open_proof(n, log2_c, evals, point, values_o, blob)
    pcs = bg.Basefold.setup(bg.BasefoldConfig(bg.BinaryReedSolomonCode(128, log2_c, n)))
    for top_nodes, subtree_log, tail_log in [(512, 16, 8), (64, 10, 9), (128, 20, 1), (4096, 12, 10)]:
        pcs.tune = dict(top_nodes=top_nodes, subtree_log=subtree_log, tail_log=tail_log)
        comm = pcs.commit(evals)
        assert comm.root == root_o, (top_nodes, subtree_log)
        values = pcs.eval(pcs.data(comm), point)
        assert np.array_equal(values, values_o)
        got = pcs.open(comm, [bg.PolyEvals(values, point)], bg.GenericChallenger.from_state(blob))
        assert got == want, (top_nodes, subtree_log, tail_log)
