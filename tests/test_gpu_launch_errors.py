"""A launch that the runtime refuses is its own call's error and nobody else's: an
evaluation queued on a stream whose capture has been invalidated fails, and the next
calls of the same thread work.  And an evaluation may be captured: a replayed graph
gives the value of the data that is there at the replay."""
import ctypes as C

import numpy as np
import pytest

from oracle import oracle as O
from basefold_gpu import rand

pytestmark = pytest.mark.gpu

RELAXED = 2  # CU_STREAM_CAPTURE_MODE_RELAXED


@pytest.fixture(scope="module")
def driver():
    import torch

    torch.zeros(1, device="cuda")  # the primary context
    cu = C.CDLL("libcuda.so.1")
    cu.cuStreamBeginCapture_v2.argtypes = [C.c_void_p, C.c_int]
    cu.cuStreamSynchronize.argtypes = [C.c_void_p]
    cu.cuStreamEndCapture.argtypes = [C.c_void_p, C.POINTER(C.c_void_p)]
    cu.cuGraphInstantiateWithFlags.argtypes = [C.POINTER(C.c_void_p), C.c_void_p, C.c_ulonglong]
    cu.cuGraphLaunch.argtypes = [C.c_void_p, C.c_void_p]
    cu.cuGraphExecDestroy.argtypes = cu.cuGraphDestroy.argtypes = [C.c_void_p]
    return cu


def _eval(lib, dev, n, point, out, stream):
    return lib.bf_eval_noalloc(C.c_void_p(dev.data_ptr()), n, C.c_void_p(point.ctypes.data), C.c_void_p(out.data_ptr()),
                               C.c_void_p(stream.cuda_stream))


def test_a_refused_launch_does_not_fail_the_next_call(built_lib, driver):
    import torch
    from basefold_gpu import _native

    bg, n = built_lib, 6
    data = rand.random_elems((1 << n) + n, 7300)
    evals, point = data[: 1 << n], np.ascontiguousarray(data[1 << n:])
    dev, out = torch.from_numpy(evals).cuda(), torch.zeros(16, dtype=torch.uint8, device="cuda")
    pcs = bg.Basefold.setup(bg.BasefoldConfig(bg.BinaryReedSolomonCode(128, 1, n)), device=0)
    st = torch.cuda.Stream()
    torch.cuda.synchronize()
    assert _eval(_native.lib(), dev, n, point, out, st) == 0  # looks the scratch up
    st.synchronize()
    assert driver.cuStreamBeginCapture_v2(st.cuda_stream, RELAXED) == 0
    assert driver.cuStreamSynchronize(st.cuda_stream) != 0  # not allowed: invalidates the capture
    refused = _eval(_native.lib(), dev, n, point, out, st)
    graph = C.c_void_p()
    assert driver.cuStreamEndCapture(st.cuda_stream, C.byref(graph)) != 0
    assert refused == _native.BF_ERR_CUDA
    assert pcs.commit(evals).root == O.commit_root(n, 1, evals)
    assert np.array_equal(pcs.eval(evals, point), O.eval_poly(n, evals, point))


@pytest.mark.parametrize("n", [1, 5, 13, 14, 17])
def test_a_captured_evaluation_replays_on_new_data(built_lib, driver, n):
    import torch
    from basefold_gpu import _native

    data = rand.random_elems((3 << n) + n, 7400 + n).reshape(-1, 16)
    point = np.ascontiguousarray(data[3 << n:])
    dev, out = torch.from_numpy(data[: 1 << n].copy()).cuda(), torch.zeros(16, dtype=torch.uint8, device="cuda")
    st = torch.cuda.Stream()
    torch.cuda.synchronize()
    assert _eval(_native.lib(), dev, n, point, out, st) == 0
    st.synchronize()
    graph, run = C.c_void_p(), C.c_void_p()
    assert driver.cuStreamBeginCapture_v2(st.cuda_stream, RELAXED) == 0
    queued = _eval(_native.lib(), dev, n, point, out, st)
    assert driver.cuStreamEndCapture(st.cuda_stream, C.byref(graph)) == 0
    assert queued == 0
    assert driver.cuGraphInstantiateWithFlags(C.byref(run), graph, 0) == 0
    for k in (1, 2):
        evals = data[k << n: (k + 1) << n]
        dev.copy_(torch.from_numpy(evals.copy()))
        out.zero_()
        torch.cuda.synchronize()
        assert driver.cuGraphLaunch(run, st.cuda_stream) == 0
        st.synchronize()
        assert np.array_equal(out.cpu().numpy().reshape(1, 16), O.eval_poly(n, evals, point))
    assert driver.cuGraphExecDestroy(run) == 0 and driver.cuGraphDestroy(graph) == 0
