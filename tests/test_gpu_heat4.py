"""FP32 Heat swept passes four levels at a time (csrc/swept_heat.cuh) against the
oracle, bit for bit: the narrowest and widest tiles that take that path (768 cells
and more on any domain, narrower ones on domains of two tiles per SM) and
widths that do not, one to several tiles (the wrapping phase-1 tile
holds both ends of the domain), insulated and periodic ends, infinities (which spread and stay), subnormals."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

HEAT, SWEPT, TIME_STEPS = 0, 1, 1


def _ic(n, seed):
    rng = np.random.default_rng(seed)
    return (50 + 40 * np.cos(2 * np.pi * 3 * np.arange(n) / n) + 4 * rng.standard_normal(n)).astype(np.float32)


def _check(sw, solver, oracle, ic, tpb, bc, steps):
    nx = ic.size
    c = oracle.reference_consts(HEAT, 4, nx, 0.004)
    c.bc = bc
    cfg = sw.make_config(HEAT, 4, alg=SWEPT, nx=nx, tpb=tpb, dt=0.004, bc=bc, time_mode=TIME_STEPS, n_steps=steps)
    want = oracle.classic(c, ic, steps)
    np.testing.assert_array_equal(solver.run(cfg, ic)[0], want, err_msg="steps %d" % steps)
    return want


@pytest.mark.parametrize("bc", [1, 2])
@pytest.mark.parametrize("tpb", [32, 64, 96, 128, 160, 224, 256, 288, 384, 512, 640, 768, 992, 1024])
@pytest.mark.parametrize("tiles", [1, 2, 3, 37])
def test_equal_the_oracle(sw, solver, oracle, tpb, tiles, bc):
    ic = _ic(tpb * tiles, tpb + tiles)
    for steps in (tpb // 2, 3 * (tpb // 2)):
        _check(sw, solver, oracle, ic, tpb, bc, steps)


@pytest.mark.parametrize("bc", [1, 2])
@pytest.mark.parametrize("tpb", [192, 224, 256, 512])
def test_narrower_tiles_on_larger_domains(sw, solver, oracle, tpb, bc):
    torch = pytest.importorskip("torch")
    tiles = 2 * torch.cuda.get_device_properties(0).multi_processor_count + 1
    _check(sw, solver, oracle, _ic(tpb * tiles, tpb), tpb, bc, 3 * (tpb // 2))


@pytest.mark.parametrize("bc", [1, 2])
def test_extreme_values(sw, solver, oracle, bc):
    ic = _ic(1024 * 5, 4)
    ic[100:104] = [0.0, -0.0, 1e-42, -1e-42]
    ic[2000], ic[3000] = 3e38, np.inf
    want = _check(sw, solver, oracle, ic, 1024, bc, 512)
    assert np.isinf(want).any() and not np.isinf(want).all()
