"""The steps left over after a swept run's whole cycles, taken in narrower cycles
and then classic steps: equal to the oracle bit for bit for every number of
steps that changes the sequence of widths, in runs, ensembles and the
no-allocation entry point, and the launches sw_plan states."""
import importlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

HEAT, KS, EULER = 0, 1, 2
SWEPT, VARIANT, TIME_STEPS = 1, 2, 1
ens = importlib.import_module("1dsweptcuda_gb300.ensemble")


def _ic(problem, prec, n, seed):
    rng = np.random.default_rng(seed)
    x = np.arange(n)
    u = np.cos(2 * np.pi * 3 * x / n) + 0.1 * rng.standard_normal(n)
    return (50 + 40 * u if problem == HEAT else u).astype(np.float64 if prec == 8 else np.float32)


def _consts(oracle, problem, prec, n, dt, bc):
    c = oracle.reference_consts(problem, prec, n, dt)
    if bc:
        c.bc = bc
    return c


@pytest.mark.parametrize("problem, prec, bc", [(HEAT, 4, 1), (HEAT, 4, 2), (HEAT, 8, 1), (KS, 4, 0), (KS, 8, 0)])
@pytest.mark.parametrize("tpb, tiles", [(1024, 5), (384, 3), (320, 7), (128, 9), (96, 4)])
def test_runs(sw, solver, oracle, problem, prec, bc, tpb, tiles):
    nx, dt = tpb * tiles, 0.004 if problem == HEAT else 0.005
    ic = _ic(problem, prec, nx, tpb)
    cycle = tpb // 2 if problem == HEAT else tpb // 8
    for steps in (cycle - 1, cycle + cycle // 2 + 1, 2 * cycle + cycle // 4, 5):
        want = oracle.classic(_consts(oracle, problem, prec, nx, dt, bc), ic, steps)
        for alg in (SWEPT, VARIANT) if problem == HEAT else (SWEPT,):
            cfg = sw.make_config(problem, prec, alg=alg, nx=nx, tpb=tpb, dt=dt, bc=bc, time_mode=TIME_STEPS, n_steps=steps)
            got, res, _ = solver.run(cfg, ic)
            np.testing.assert_array_equal(got, want, err_msg="alg %d steps %d" % (alg, steps))
            assert res.n_steps == steps and res.tile == tpb
            if res.launches:
                assert res.launches == sw.plan(cfg)[0].launches


@pytest.mark.parametrize("problem, prec", [(HEAT, 4), (HEAT, 8), (KS, 4)])
@pytest.mark.parametrize("alg", [SWEPT, VARIANT])
def test_ensembles(sw, solver, oracle, problem, prec, alg):
    tpb = 512
    nx = tpb * np.array([1, 3, 2, 7, 1], dtype=np.int64)
    dt = 0.004 if problem == HEAT else 0.005
    ic = np.concatenate([_ic(problem, prec, int(n), i) for i, n in enumerate(nx)])
    cycle = tpb // 2 if problem == HEAT else tpb // 8
    for steps in (cycle - 1, cycle + cycle // 2 + cycle // 8 + 3):
        cfg = sw.make_config(problem, prec, alg=alg, tpb=tpb, dt=dt, time_mode=TIME_STEPS, n_steps=steps)
        got, _ = solver.run_batch(cfg, nx, ic)
        want = ens.concat([oracle.classic(_consts(oracle, problem, prec, int(n), dt, 0), part, steps)
                           for part, n in zip(ens.split(ic, nx, 1), nx)])
        np.testing.assert_array_equal(got, want)


def test_no_allocation(sw, oracle):
    torch = pytest.importorskip("torch")
    nx, tpb, dt, steps = 4096, 512, 0.005, 64 + 32 + 16 + 3
    ic = _ic(KS, 4, nx, 2)
    u = torch.from_numpy(ic.copy()).cuda()
    cfg = sw.make_config(KS, 4, alg=SWEPT, nx=nx, tpb=tpb, dt=dt, time_mode=TIME_STEPS, n_steps=steps)
    sw.native.run_device_noalloc(cfg, u.data_ptr(), sw.native.torch_stream())
    torch.cuda.synchronize()
    np.testing.assert_array_equal(u.cpu().numpy(), oracle.classic(oracle.reference_consts(KS, 4, nx, dt), ic, steps))
