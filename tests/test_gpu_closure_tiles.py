"""The closure's forward kernels at the edges of their tiles: domains of 128
cells (one tile that wraps onto itself), of a few tiles with a short last one,
and of more tiles than there are resident blocks; the plain coarse step at the
same sizes, from buffers that are only 4-byte aligned."""
import importlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

SIZES = [(1, 128), (5, 128), (3, 256), (2, 384), (1, 1152), (1300, 128), (700, 256)]


@pytest.fixture(scope="module")
def cl():
    return importlib.import_module("1dsweptcuda_gb300.closure")


def _theta(seed):
    rng = np.random.default_rng(seed)
    return np.concatenate([rng.standard_normal(160) * np.sqrt(2 / 5), rng.standard_normal(32) * 0.1,
                           rng.standard_normal(5120) * np.sqrt(2 / 160), rng.standard_normal(32) * 0.1,
                           rng.standard_normal(160) * 0.1, [0.05], [0.5]]).astype(np.float32)


@pytest.mark.parametrize("n_dom,n", SIZES)
def test_infer_matches_oracle(sw, solver, cl, n_dom, n):
    # the activations' rounding to BF16 and the SFU's tanh (relative 2^-10.7) bound the error as at any size
    from oracle import closure as ocl
    rng = np.random.default_rng(n_dom + n)
    u = (rng.standard_normal((n_dom, n)) * 1.5).astype(np.float32)
    th = _theta(n)
    got = cl.Closure(solver, th).infer(torch.from_numpy(u).cuda()).cpu().numpy().astype(np.float64)
    rows = np.unique(np.linspace(0, n_dom - 1, min(n_dom, 40)).astype(int))
    want = ocl.forward(th.astype(np.float64), u[rows].astype(np.float64))
    assert np.abs(got[rows] - want).max() / np.abs(want).max() < 5e-3


@pytest.mark.parametrize("n_dom,n", SIZES)
def test_step_is_the_classic_step_plus_the_correction(sw, solver, cl, n_dom, n):
    rng = np.random.default_rng(n_dom * n)
    u = torch.from_numpy(rng.standard_normal((n_dom, n)).astype(np.float32)).cuda()
    c = cl.Closure(solver, _theta(7))
    plain, both = u.clone(), u.clone()
    c.step(plain, 1, use_closure=False)
    c.step(both, 1, use_closure=True)
    assert torch.equal(both, plain + c.infer(u))
    cfg = sw.make_config(sw.KS, 4, alg=sw.ALG_CLASSIC, tpb=128, dt=cl.COARSE_DT, dx=cl.COARSE_DX,
                         time_mode=sw.TIME_STEPS, n_steps=1)
    want, _ = solver.run_batch(cfg, np.full(n_dom, n, dtype=np.int64), u.cpu().numpy().ravel())
    np.testing.assert_array_equal(plain.cpu().numpy().ravel(), want)


@pytest.mark.parametrize("use_closure", [False, True])
def test_several_steps_from_an_unaligned_buffer(sw, solver, cl, use_closure):
    rng = np.random.default_rng(3)
    u = torch.from_numpy(rng.standard_normal((4, 384)).astype(np.float32)).cuda()
    c = cl.Closure(solver, _theta(8))
    shifted = torch.zeros(4 * 384 + 1, dtype=torch.float32, device="cuda")[1:].view(4, 384)
    shifted.copy_(u)
    one = u.clone()
    c.step(shifted, 5, use_closure=use_closure)
    for _ in range(5):
        c.step(one, 1, use_closure=use_closure)
    assert torch.equal(shifted, one)
