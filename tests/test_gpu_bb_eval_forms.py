"""BabyBear column evaluations with four columns a lane (rows of whole 16-byte groups,
128 columns or more, aligned data) and with one: widths on both sides of each
condition, row counts around a warp's and a block's share, data that starts off
a 16-byte boundary, and rows of words that are not canonical (taken mod p)."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w", [124, 126, 127, 128, 130, 132, 256, 300])
def test_column_evaluations(built_lib, w):
    from basefold_gpu import BasefoldConfig, prime
    import torch

    for n in (1, 3, 6, 10):
        rng = np.random.default_rng(1000 * n + w)
        data = rng.integers(0, O.BB_P, size=(1 << n, w), dtype=np.uint64).astype(np.uint32)
        data[0] = O.BB_P - 1
        data[-1, ::3] = 0
        point = rng.integers(0, O.BB_P, size=(n, 5), dtype=np.uint32)
        pcs = prime.BabyBearBasefold.setup(BasefoldConfig(prime.ReedSolomonCode(128, 1, n)), device=0)
        want = np.asarray(O.bb_harness_prepare(n, 1, data, point)[1]).reshape(-1, 5)
        assert np.array_equal(pcs.eval(pcs.commit(data), point), want), n
        raw = data.astype(np.uint64) + np.uint64(O.BB_P) * rng.integers(0, 2, size=data.shape, dtype=np.uint64)
        raw[0] = 2 * O.BB_P + 7  # the largest multiple of p below 2^32, and a bit
        shifted = data.copy()
        shifted[0] = 7
        want_raw = np.asarray(O.bb_harness_prepare(n, 1, shifted, point)[1]).reshape(-1, 5)
        flat = raw.astype(np.uint32).reshape(-1)
        for off in (0, 1):
            buf = torch.from_numpy(np.concatenate([np.zeros(off, np.uint32), flat]).view(np.int32)).cuda()
            torch.cuda.synchronize()
            assert np.array_equal(pcs.eval_device(buf.data_ptr() + 4 * off, point, w), want_raw), (n, off)
