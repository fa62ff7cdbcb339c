"""Batched verify of proofs that someone else keeps writing: an opened row, the
final polynomial or a folded-codeword root flips between its honest value and
another one while batches run.  Each value is taken once, so every code is one that
a proof at rest can have: a wrong row fails its path (never the fold alone), a wrong
final polynomial or root fails the final check (never a query)."""
import ctypes as C
import threading

import numpy as np
import pytest

from oracle import oracle as O
from basefold_gpu import rand

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w", [1, 3])
@pytest.mark.parametrize("part", ["row", "final", "root"])
def test_changing_bytes_give_codes_of_some_proof(built_lib, part, w):
    from basefold_gpu._native import BfVerifyJob, check, lib

    bg, n, count = built_lib, 8, 6
    pcs = bg.Basefold.setup(bg.BasefoldConfig(bg.BinaryReedSolomonCode(128, 1, n)), device=0)
    data = rand.random_elems((w << n) + n, 6300 + w)
    evals, point = data[: w << n], np.ascontiguousarray(data[w << n:])
    root, values, blob = O.harness_prepare(n, 1, evals, point, width=w)
    proof = O.open_proof(n, 1, evals, point, values, blob, width=w)
    # round polynomials (8 + 32 bytes each), final polynomial, roots, openings
    final = 8 + 40 * n + 8
    roots = final + 16 + 8
    row = roots + 32 * n + 8 + 8
    at = {"row": row, "final": final, "root": roots + 32 * (n - 1)}[part]
    wrong = 3 if part == "row" else 1  # the path's code; the final polynomial's

    buf = np.zeros(len(proof) + 16, np.uint8)
    lo = (-buf.ctypes.data) % 16
    buf[lo: lo + len(proof)] = np.frombuffer(proof, np.uint8)
    cell = buf[lo + at: lo + at + 16]
    honest, other = cell.copy(), cell ^ 0x5A
    rt = np.frombuffer(root, np.uint8).copy()
    vals = np.ascontiguousarray(np.asarray(values, np.uint8).reshape(-1, 16))

    def codes():
        jobs, keep = (BfVerifyJob * count)(), []
        for job in jobs:
            ch = bg.GenericChallenger.from_state(blob)
            keep.append(ch)
            job.root, job.point, job.values, job.width = rt.ctypes.data, point.ctypes.data, vals.ctypes.data, w
            job.challenger, job.proof, job.proof_len = C.cast(ch._h, C.c_void_p).value, buf.ctypes.data + lo, len(proof)
        check(lib().bf_verify_batch(pcs._h, jobs, count))
        return [j.result for j in jobs]

    assert codes() == [0] * count
    stop = threading.Event()

    def write():
        while not stop.is_set():
            cell[:] = other
            cell[:] = honest

    writer = threading.Thread(target=write)
    writer.start()
    try:
        seen = {c for _ in range(100) for c in codes()}
    finally:
        stop.set()
        writer.join()
    assert seen <= {0, wrong}
    cell[:] = other
    assert codes() == [wrong] * count
