"""Batched verify reads the proofs where the caller has them, or copies the ones
whose address is not a multiple of 8: the same codes as the oracle's for proofs at
any address, aligned and not in one batch, valid, tampered, cut short and empty,
narrow and wide."""
import ctypes as C

import numpy as np
import pytest

from oracle import oracle as O
from basefold_gpu import rand

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,w", [(0, 1), (7, 1), (10, 1), (6, 3)])
def test_proofs_at_any_address(built_lib, n, w):
    from basefold_gpu._native import BfVerifyJob, check, lib

    bg = built_lib
    pcs = bg.Basefold.setup(bg.BasefoldConfig(bg.BinaryReedSolomonCode(128, 1, n)), device=0)
    data = rand.random_elems((w << n) + n, 5200 + n)
    evals, point = data[: w << n], np.ascontiguousarray(data[w << n:])
    root, values, blob = O.harness_prepare(n, 1, evals, point, width=w)
    proof = O.open_proof(n, 1, evals, point, values, blob, width=w)
    bad = bytearray(proof)
    bad[-20] ^= 1
    proofs = [proof, bytes(bad), proof[:-8], b"", proof]
    cases = [(p, shift) for p in proofs for shift in (0, 1, 4, 8, 13)]
    jobs = (BfVerifyJob * len(cases))()
    rt = np.frombuffer(root, np.uint8).copy()
    vals = np.ascontiguousarray(np.asarray(values, np.uint8).reshape(-1, 16))
    pt = point if n else np.zeros((1, 16), np.uint8)
    keep = []
    for job, (p, shift) in zip(jobs, cases):
        buf = np.zeros(len(p) + 64, np.uint8)
        at = (-buf.ctypes.data) % 16 + shift
        buf[at: at + len(p)] = np.frombuffer(p, np.uint8)
        ch = bg.GenericChallenger.from_state(blob)
        keep += [buf, ch]
        job.root, job.point, job.values, job.width = rt.ctypes.data, pt.ctypes.data, vals.ctypes.data, w
        job.challenger, job.proof, job.proof_len = C.cast(ch._h, C.c_void_p).value, buf.ctypes.data + at, len(p)
    check(lib().bf_verify_batch(pcs._h, jobs, len(cases)))
    want = {p: O.verify(n, 1, root, point, values, blob, p, width=w) for p in set(proofs)}
    assert [j.result for j in jobs] == [want[p] for p, _ in cases]
    assert want[proof] == 0 and want[bytes(bad)] != 0
