"""The prime-field open around the sizes where its last rounds move into one
block (folds of 2^8 outputs): opens that run wholly in the block, enter it in the
first round with base-field data, or after some launched rounds.
Whole proofs against the oracle's bytes."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _rnd(shape, seed, lo=0):
    return np.random.default_rng(seed).integers(lo, O.BB_P, size=shape, dtype=np.uint64).astype(np.uint32)


@pytest.mark.parametrize("w", [1, 3])
@pytest.mark.parametrize("n,log2_c", [(1, 1), (6, 1), (7, 1), (8, 1), (9, 1), (11, 1), (5, 3), (6, 3), (8, 0), (9, 0), (10, 2)])
def test_reed_solomon_open_around_the_tail(built_lib, n, log2_c, w):
    from basefold_gpu import BasefoldConfig, GenericChallenger, prime

    data, point = _rnd((1 << n, w), 100 * n + log2_c), _rnd((n, 5), 200 * n + w)
    pcs = prime.BabyBearBasefold.setup(BasefoldConfig(prime.ReedSolomonCode(128, log2_c, n)), device=0)
    comm = pcs.commit(data)
    root, values, blob = O.bb_harness_prepare(n, log2_c, data if w > 1 else data.reshape(-1), point)
    assert comm.root == root
    # a transcript with a long, odd-length past: the first round absorbs blocks
    # and appends at an unaligned position
    for past in (b"", bytes(range(133)), bytes(307)):
        ch = GenericChallenger.from_state(blob)
        ch.observe(past)
        before = ch.state()
        proof = pcs.open(comm, [prime.PrimePolyEvals(values, point)], ch)
        assert proof == O.bb_open(n, log2_c, data if w > 1 else data.reshape(-1), point, values, before)
