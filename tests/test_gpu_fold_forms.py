"""Open rounds at the sizes where a fold changes form: one thread per output and
a pair of lanes per leaf hash up to 2^17 leaves (binary) and 2^13 (BabyBear), one
thread per leaf above; and the commits whose last-pass tiles have fewer pairs than
threads.  Whole proofs against the oracle's bytes."""
import numpy as np
import pytest

from oracle import oracle as O
from basefold_gpu import rand

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,log2_c", [(12, 1), (14, 1), (16, 3), (18, 1)])
def test_binary_folds(built_lib, n, log2_c):
    bg = built_lib
    data = rand.random_elems((1 << n) + n, 9900 + n)
    evals, point = data[: 1 << n], data[1 << n:]
    root_o, values_o, blob = O.harness_prepare(n, log2_c, evals, point)
    pcs = bg.Basefold.setup(bg.BasefoldConfig(bg.BinaryReedSolomonCode(128, log2_c, n)))
    comm = pcs.commit(evals)
    assert comm.root == root_o
    values = pcs.eval(pcs.data(comm), point)
    assert np.array_equal(values, values_o)
    got = pcs.open(comm, [bg.PolyEvals(values, point)], bg.GenericChallenger.from_state(blob))
    assert got == O.open_proof(n, log2_c, evals, point, values_o, blob)


@pytest.mark.parametrize("n,log2_c,w", [(12, 1, 1), (13, 1, 2), (14, 1, 1), (13, 2, 3)])
def test_prime_folds(built_lib, n, log2_c, w):
    from basefold_gpu import BasefoldConfig, GenericChallenger, prime

    rng = np.random.default_rng(9950 + n + w)
    data = rng.integers(0, O.BB_P, (1 << n, w), dtype=np.uint32)
    point = rng.integers(0, O.BB_P, (n, 5), dtype=np.uint32)
    flat = data if w > 1 else data.reshape(-1)
    pcs = prime.BabyBearBasefold.setup(BasefoldConfig(prime.ReedSolomonCode(128, log2_c, n)), device=0)
    comm = pcs.commit(data)
    root, values, blob = O.bb_harness_prepare(n, log2_c, flat, point)
    assert comm.root == root
    proof = pcs.open(comm, [prime.PrimePolyEvals(values, point)], GenericChallenger.from_state(blob))
    assert proof == O.bb_open(n, log2_c, flat, point, values, blob)


@pytest.mark.parametrize("n,log2_c,lk,w", [(11, 0, 9, 1), (12, 1, 9, 2), (14, 0, 10, 1)])
def test_prime_folds_without_a_tail(built_lib, n, log2_c, lk, w):
    """Base codes of more than 2^8 rows: the last round's fix is a launch of its
    own after rounds that fix in the fold's."""
    from basefold_gpu import BasefoldConfig, GenericChallenger, prime

    rng = np.random.default_rng(9970 + n + w)
    data = rng.integers(0, O.BB_P, (1 << n, w), dtype=np.uint32)
    point = rng.integers(0, O.BB_P, (n, 5), dtype=np.uint32)
    flat = data if w > 1 else data.reshape(-1)
    kw = dict(log2_k0=lk, ts=O.bb_random_ts(n, log2_c, lk, 5))
    code = prime.GenericRandomFoldableCode(128, log2_c, lk, n - lk, kw["ts"])
    pcs = prime.BabyBearBasefold.setup(BasefoldConfig(code), device=0)
    comm = pcs.commit(data)
    root, values, blob = O.bb_harness_prepare(n, log2_c, flat, point, **kw)
    assert comm.root == root
    proof = pcs.open(comm, [prime.PrimePolyEvals(values, point)], GenericChallenger.from_state(blob))
    assert proof == O.bb_open(n, log2_c, flat, point, values, blob, **kw)
