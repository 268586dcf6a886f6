"""Euler FP64 forms its quotients and square roots on the integer pipe where
their operands are normal numbers with a normal result, and on the FP64 pipe
where they are not: states scaled so that products, quotients and pressure
differences leave that range (and overflow) in some cells or all, against the
oracle, bit for bit (any NaN for a NaN)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EULER, TIME_STEPS = 2, 1


def _same(a, b):
    nan = np.isnan(a) & np.isnan(b)
    return bool(((a.view(np.int64) == b.view(np.int64)) | nan).all())


@pytest.mark.parametrize("alg", [0, 1, 2])
@pytest.mark.parametrize("scale", [1e-320, 1e-160, 1e-104, 1e103, 1e160])
@pytest.mark.parametrize("everywhere", [True, False])
def test_euler_operands_outside_the_integer_range(sw, solver, oracle, alg, scale, everywhere):
    nx, tpb, steps = 2048, 128, 2 * 32 + 3
    dt = 0.1 / (nx - 2)
    rng = np.random.default_rng(17)
    rho, u, p = 0.5 + rng.random(nx), 0.2 * rng.standard_normal(nx), 0.3 + rng.random(nx)
    ic = np.stack([rho, rho * u, p / 0.4 + 0.5 * rho * u * u], 1)
    if everywhere:
        ic[1:-1] *= scale
    else:
        ic[700:713] *= scale
        ic[1500] *= scale
    ic[0], ic[-1] = oracle.reference_ic(EULER, 8, nx).reshape(-1, 3)[[0, -1]]
    ic = ic.ravel().copy()
    want = oracle.classic(oracle.reference_consts(EULER, 8, nx, dt), ic, steps)
    cfg = sw.make_config(EULER, 8, alg=alg, nx=nx, tpb=tpb, dt=dt, time_mode=TIME_STEPS, n_steps=steps)
    got, _, _ = solver.run(cfg, ic)
    assert _same(got, want)
