"""FP32 classic Heat and KS with four cells per thread against the oracle, bit for
bit: the smallest domain, partial blocks, a state that is not 16-byte aligned
(one cell per thread), both Heat boundaries, long chains of dependent launches,
and ensembles whose lengths are, or are not, all multiples of four."""
import importlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

HEAT, KS, CLASSIC, TIME_STEPS = 0, 1, 0, 1
ens = importlib.import_module("1dsweptcuda_gb300.ensemble")


def _ic(problem, n, seed):
    rng = np.random.default_rng(seed)
    x = np.arange(n)
    u = np.cos(2 * np.pi * 3 * x / n) + 0.1 * rng.standard_normal(n)
    return (50 + 40 * u if problem == HEAT else u).astype(np.float32)


def _consts(oracle, problem, n, dt, bc):
    c = oracle.reference_consts(problem, 4, n, dt)
    if bc is not None:
        c.bc = bc
    return c


@pytest.mark.parametrize("problem, bc", [(HEAT, 1), (HEAT, 2), (KS, 2)])
@pytest.mark.parametrize("nx", [32, 1024, 1056, 9984])
@pytest.mark.parametrize("offset", [0, 1, 2, 4])
def test_single_domain(sw, solver, oracle, problem, bc, nx, offset):
    torch = pytest.importorskip("torch")
    dt, steps = (0.004, 301) if problem == HEAT else (0.005, 150)
    ic = _ic(problem, nx, nx + offset)
    buf = torch.zeros(nx + 8, dtype=torch.float32, device="cuda")
    u = buf[offset:offset + nx]
    u.copy_(torch.from_numpy(ic))
    cfg = sw.make_config(problem, 4, alg=CLASSIC, nx=nx, tpb=32, dt=dt, bc=bc, time_mode=TIME_STEPS, n_steps=steps)
    solver.run_device(cfg, u.data_ptr(), sw.native.torch_stream())
    want = oracle.classic(_consts(oracle, problem, nx, dt, oracle.BC_PERIODIC if problem == HEAT and bc == 2 else None), ic, steps)
    np.testing.assert_array_equal(u.cpu().numpy(), want)
    rest = torch.cat([buf[:offset], buf[offset + nx:]])
    assert not rest.any()


@pytest.mark.parametrize("lengths", [[32, 36, 1028, 4, 260] * 3, [33, 47, 1030, 65, 129]])
@pytest.mark.parametrize("problem", [HEAT, KS])
def test_ensemble(sw, solver, oracle, problem, lengths):
    nx = np.maximum(np.array(lengths, dtype=np.int64), 32)
    dt, steps = (0.004, 51) if problem == HEAT else (0.005, 40)
    ic = np.concatenate([_ic(problem, int(n), i) for i, n in enumerate(nx)])
    cfg = sw.make_config(problem, 4, alg=CLASSIC, dt=dt, time_mode=TIME_STEPS, n_steps=steps)
    got, _ = solver.run_batch(cfg, nx, ic)
    want = ens.concat([oracle.classic(_consts(oracle, problem, int(n), dt, None), part, steps)
                       for part, n in zip(ens.split(ic, nx, 1), nx)])
    np.testing.assert_array_equal(got, want)
