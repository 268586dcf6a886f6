"""A launch that fails reports its error once: the call returns it, and the
thread's last CUDA error is clear again, so that the next call (of this library
or of torch, which share the runtime) does not report it a second time.  The
launch fails on the host: its stream's capture has been invalidated."""
import ctypes as C

import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

CAPTURE_RELAXED = 2


@pytest.mark.parametrize("problem, prec, tpb", [(0, 4, 1024), (0, 8, 128), (1, 4, 256), (1, 8, 256), (2, 8, 128)])
def test_a_failed_launch_leaves_no_last_error(sw, problem, prec, tpb):
    lib = sw.library()
    rt = C.CDLL("libcudart.so.13")  # the runtime the library is linked to, already loaded
    cells = 2 * tpb
    cfg = sw.make_config(problem, prec, alg=sw.ALG_SWEPT, nx=cells, tpb=tpb, dt=1e-4, time_mode=sw.TIME_STEPS, n_steps=tpb)
    u = torch.ones(cells * (4 if problem == 2 else 1), dtype=torch.float64 if prec == 8 else torch.float32, device="cuda")
    sw.native.run_device_noalloc(cfg, u.data_ptr(), sw.native.torch_stream())  # the first call looks the scratch up
    torch.cuda.synchronize()
    stream = torch.cuda.Stream()
    s = C.c_void_p(stream.cuda_stream)
    assert rt.cudaStreamBeginCapture(s, CAPTURE_RELAXED) == 0
    try:
        assert rt.cudaStreamSynchronize(s) != 0  # not allowed in a capture: invalidates it
        rt.cudaGetLastError()
        rc = lib.sw_run_device_noalloc(C.byref(cfg), C.c_void_p(u.data_ptr()), s)
        left = rt.cudaPeekAtLastError()
    finally:
        graph = C.c_void_p()
        rt.cudaStreamEndCapture(s, C.byref(graph))
        rt.cudaGetLastError()
    assert rc == -4  # SW_ERR_CUDA
    assert left == 0
    sw.native.run_device_noalloc(cfg, u.data_ptr(), sw.native.torch_stream())
    torch.cuda.synchronize()
