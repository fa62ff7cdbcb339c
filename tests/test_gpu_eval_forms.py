"""The evaluation of one polynomial at every size where its form or its split into
two eq tables changes, from device and host data, at points with coordinates 0 and
1 among uniform ones and at any host address; and the eq table of the open, in one
launch up to 16 variables and from two tables above.  Against the oracle's values
and proofs."""
import ctypes as C

import numpy as np
import pytest

from oracle import oracle as O
from basefold_gpu import rand

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", list(range(0, 13)) + [15, 16, 17, 19])
def test_values_match_the_oracle(built_lib, n):
    from basefold_gpu._native import check, lib

    bg = built_lib
    data = rand.random_elems((1 << n) + n, 6600 + n)
    evals, point = data[: 1 << n], np.ascontiguousarray(data[1 << n:])
    if n >= 3:
        point[0] = 0
        point[n // 2] = np.frombuffer((1 | 0xc2 << 120).to_bytes(16, "little"), np.uint8)  # the field's one
    pcs = bg.Basefold.setup(bg.BasefoldConfig(bg.BinaryReedSolomonCode(128, 1, n)), device=0)
    want = O.eval_poly(n, evals, point)
    comm = pcs.commit(evals)
    for shift in (0, 1, 8):
        buf = np.zeros(16 * n + 64, np.uint8)
        at = (-buf.ctypes.data) % 16 + shift
        buf[at: at + 16 * n] = point.reshape(-1)
        out = np.zeros((1, 16), np.uint8)
        check(lib().bf_eval(pcs._h, comm._h, C.c_void_p(buf.ctypes.data + at), C.c_void_p(out.ctypes.data)))
        assert np.array_equal(out, want), shift
    assert np.array_equal(pcs.eval(evals, point if n else np.zeros((0, 16), np.uint8)), want)


@pytest.mark.parametrize("n", [2, 6, 16, 17, 18])
def test_opens_with_every_eq_table_form(built_lib, n):
    bg = built_lib
    data = rand.random_elems((1 << n) + n, 6700 + n)
    evals, point = data[: 1 << n], data[1 << n:]
    root, values, blob = O.harness_prepare(n, 1, evals, point)
    pcs = bg.Basefold.setup(bg.BasefoldConfig(bg.BinaryReedSolomonCode(128, 1, n)), device=0)
    comm = pcs.commit(evals)
    got = pcs.open(comm, [bg.PolyEvals(values, point)], bg.GenericChallenger.from_state(blob))
    assert got == O.open_proof(n, 1, evals, point, values, blob)
