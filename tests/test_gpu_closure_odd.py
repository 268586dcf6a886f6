"""The closure's forward kernel with two tiles per block on an odd number of
tiles: the last block's second half has no tile.  Tiles of 124 outputs (128 in
domains of 128 cells), two at a time above three per SM; with five blocks per SM
the last size takes each block through several rounds of its stride."""
import importlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

SIZES = [(1301, 128), (701, 256), (691, 1024)]  # 1301, 2103 and 6219 tiles


@pytest.fixture(scope="module")
def cl():
    return importlib.import_module("1dsweptcuda_gb300.closure")


def _closure(cl, solver, seed):
    rng = np.random.default_rng(seed)
    theta = np.concatenate([rng.standard_normal(160) * np.sqrt(2 / 5), rng.standard_normal(32) * 0.1,
                            rng.standard_normal(5120) * np.sqrt(2 / 160), rng.standard_normal(32) * 0.1,
                            rng.standard_normal(160) * 0.1, [0.05], [0.5]]).astype(np.float32)
    return cl.Closure(solver, theta), theta


@pytest.mark.parametrize("n_dom, n", SIZES)
def test_infer(sw, solver, cl, n_dom, n):
    from oracle import closure as ocl
    c, theta = _closure(cl, solver, n)
    u = torch.from_numpy((np.random.default_rng(n_dom).standard_normal((n_dom, n)) * 1.5).astype(np.float32)).cuda()
    got = c.infer(u)
    # the same arithmetic row for row in the one-tile kernel, which a few domains take
    for d in (0, 1, n_dom // 2, n_dom - 2, n_dom - 1):
        assert torch.equal(got[d], c.infer(u[d:d + 1].clone())[0]), d
    # the activations' rounding to BF16 and the SFU's tanh (relative 2^-10.7) bound the error as at any size
    last = slice(n_dom - 2, n_dom)
    want = ocl.forward(theta.astype(np.float64), u[last].cpu().numpy().astype(np.float64))
    assert np.abs(got[last].cpu().numpy().astype(np.float64) - want).max() / np.abs(want).max() < 5e-3


@pytest.mark.parametrize("n_dom, n", SIZES)
def test_step(sw, solver, cl, n_dom, n):
    c, _ = _closure(cl, solver, 7)
    u = torch.from_numpy(np.random.default_rng(n_dom * n).standard_normal((n_dom, n)).astype(np.float32)).cuda()
    plain, both = u.clone(), u.clone()
    c.step(plain, 1, use_closure=False)
    c.step(both, 1, use_closure=True)
    assert torch.equal(both, plain + c.infer(u))
    several, one = u.clone(), u.clone()  # dependent launches
    c.step(several, 3, use_closure=True)
    for _ in range(3):
        c.step(one, 1, use_closure=True)
    assert torch.equal(several, one)
