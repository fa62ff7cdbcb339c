"""Opens whose first round takes the fold of one thread per leaf (above 2^17 leaves,
binary, or 2^13, BabyBear, where the fix runs on a second stream) and whose later
rounds take the small form; and host commits of one large polynomial, whose first
column pass runs slice by slice, against the same data committed from the device."""
import numpy as np
import pytest

from oracle import oracle as O
from basefold_gpu import rand

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,log2_c", [(19, 1), (17, 3)])
def test_binary_open_from_the_large_fold_to_the_small(built_lib, n, log2_c):
    bg = built_lib
    data = rand.random_elems((1 << n) + n, 9800 + n)
    evals, point = data[: 1 << n], data[1 << n:]
    root, values, blob = O.harness_prepare(n, log2_c, evals, point)
    pcs = bg.Basefold.setup(bg.BasefoldConfig(bg.BinaryReedSolomonCode(128, log2_c, n)))
    comm = pcs.commit(evals)
    assert comm.root == root
    want = O.open_proof(n, log2_c, evals, point, values, blob)
    assert pcs.open(comm, [bg.PolyEvals(values, point)], bg.GenericChallenger.from_state(blob)) == want
    session = pcs.open_session(comm, bg.PolyEvals(values, point))
    assert session.prove(bg.GenericChallenger.from_state(blob)) == want


@pytest.mark.parametrize("n,log2_c,w", [(15, 1, 1), (14, 2, 3)])
def test_prime_open_from_the_large_fold_to_the_small(built_lib, n, log2_c, w):
    from basefold_gpu import BasefoldConfig, GenericChallenger, prime

    rng = np.random.default_rng(9850 + n + w)
    data = rng.integers(0, O.BB_P, (1 << n, w), dtype=np.uint32)
    point = rng.integers(0, O.BB_P, (n, 5), dtype=np.uint32)
    flat = data if w > 1 else data.reshape(-1)
    pcs = prime.BabyBearBasefold.setup(BasefoldConfig(prime.ReedSolomonCode(128, log2_c, n)), device=0)
    comm = pcs.commit(data)
    root, values, blob = O.bb_harness_prepare(n, log2_c, flat, point)
    assert comm.root == root
    proof = pcs.open(comm, [prime.PrimePolyEvals(values, point)], GenericChallenger.from_state(blob))
    assert proof == O.bb_open(n, log2_c, flat, point, values, blob)


@pytest.mark.parametrize("n,log2_c", [(22, 1), (23, 1), (21, 2), (20, 3)])
def test_host_commits_of_large_polynomials(built_lib, n, log2_c):
    import torch

    bg = built_lib
    data = np.random.default_rng(9900 + n).integers(0, 256, (1 << n, 16), dtype=np.uint8)
    pcs = bg.Basefold.setup(bg.BasefoldConfig(bg.BinaryReedSolomonCode(128, log2_c, n)))
    dev = torch.from_numpy(data).cuda()
    torch.cuda.synchronize()
    assert pcs.commit(data).root == pcs.commit_device(dev.data_ptr(), 1, keep=dev).root
