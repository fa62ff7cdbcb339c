"""The encode's column passes: pairs of layers with shared-memory tables of the
twiddles (large for many columns per group, small for a few hundred), and the few
layers left of a wide matrix without.  Widths that fill,
straddle and miss the blocks, odd and even layer counts, every blowup, host
input in slices, and inputs whose bit groups are all zero or all one.  Roots
against the oracle (a root binds every codeword entry)."""
import numpy as np
import pytest

from oracle import oracle as O
from basefold_gpu import rand

pytestmark = pytest.mark.gpu


def _matrix(n, w, seed):
    data = rand.random_elems(w << n, seed)
    data[1::5] = 0
    data[2::9] = 255
    return data


@pytest.mark.parametrize("n,log2_c,w", [(9, 1, 1024), (10, 1, 513), (12, 1, 129), (13, 2, 33), (16, 1, 8), (18, 1, 2),
                                        (17, 1, 5), (11, 1, 300), (16, 4, 3), (12, 1, 256), (14, 1, 255)])
def test_matrix_commits_match_the_oracle(built_lib, n, log2_c, w):
    bg = built_lib
    data = _matrix(n, w, 4000 + n + w)
    pcs = bg.Basefold.setup(bg.BasefoldConfig(bg.BinaryReedSolomonCode(128, log2_c, n)))
    import torch

    dev = torch.from_numpy(data).cuda()
    torch.cuda.synchronize()
    want = O.commit_root(n, log2_c, data, width=w)
    assert pcs.commit_device(dev.data_ptr(), w, keep=dev).root == want
    assert pcs.commit(data, width=w).root == want  # host input, sliced from 2^16 rows on


@pytest.mark.parametrize("n,log2_c", [(20, 1), (21, 1), (19, 2), (18, 3)])
def test_single_polynomial_commits_match_the_oracle(built_lib, n, log2_c):
    bg = built_lib
    data = _matrix(n, 1, 4100 + n)
    pcs = bg.Basefold.setup(bg.BasefoldConfig(bg.BinaryReedSolomonCode(128, log2_c, n)))
    import torch

    dev = torch.from_numpy(data).cuda()
    torch.cuda.synchronize()
    want = O.commit_root(n, log2_c, data)
    assert pcs.commit_device(dev.data_ptr(), 1, keep=dev).root == want
    assert pcs.commit(data).root == want
