"""FP32 Heat and KS passes of the paired and the four-level kernels where the
launch covers other tiles than a whole run's: the hybrid variant (every tile but
the wrapping one, which the host computes: an odd number here, so that the last
block of pairs has one tile) and sw_swept_pass, one launch at a time.  Equal to
the classic scheme bit for bit."""
import importlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
split = importlib.import_module("1dsweptcuda_gb300.split")

HEAT, KS = 0, 1
# (problem, tpb, tiles, bc): pairs of one and two position groups per thread need more tiles than SMs and sixteen
# times as many, the four-level kernel two per SM below 768 cells
CASES = [(KS, 256, 308, 0), (KS, 768, 2434, 0), (KS, 128, 1218, 0), (HEAT, 1024, 2, 1), (HEAT, 1024, 6, 2),
         (HEAT, 768, 4, 1), (HEAT, 256, 308, 1), (HEAT, 224, 308, 2)]


def _case(sw, problem, tpb, tiles, bc):
    nx = tpb * tiles
    dt = 0.004 if problem == HEAT else 0.005
    x = np.arange(nx)
    u = np.cos(2 * np.pi * 3 * x / nx) + 0.1 * np.random.default_rng(tpb + tiles).standard_normal(nx)
    ic = (50 + 40 * u if problem == HEAT else u).astype(np.float32)
    return sw.make_config(problem, 4, nx=nx, tpb=tpb, dt=dt, bc=bc, time_mode=sw.TIME_STEPS), ic


def _classic(sw, solver, cfg, ic, steps):
    c = sw.make_config(cfg.problem, 4, alg=sw.ALG_CLASSIC, nx=cfg.nx, tpb=32, dt=cfg.dt, bc=cfg.bc,
                       time_mode=sw.TIME_STEPS, n_steps=steps)
    return solver.run(c, ic)[0]


@pytest.mark.parametrize("problem, tpb, tiles, bc", CASES)
def test_host_tile(sw, solver, problem, tpb, tiles, bc):
    cfg, ic = _case(sw, problem, tpb, tiles, bc)
    cfg.alg, cfg.flags = sw.ALG_SWEPT, sw.FLAG_HOST_TILE
    cycle = split.steps_per_diamond(problem, tpb)
    for steps in (cycle, 2 * cycle + 3):  # down-triangles of phase 1 and 0
        cfg.n_steps = steps
        np.testing.assert_array_equal(solver.run(cfg, ic)[0], _classic(sw, solver, cfg, ic, steps))


@pytest.mark.parametrize("problem, tpb, tiles, bc", CASES)
def test_single_passes(sw, solver, problem, tpb, tiles, bc):
    cfg, ic = _case(sw, problem, tpb, tiles - 1, bc)
    cfg.alg = sw.ALG_SWEPT
    cycle = split.steps_per_diamond(problem, tpb)
    for steps in (cycle, 2 * cycle):
        u = torch.from_numpy(ic).cuda()
        slots = torch.empty(2 * ic.size, dtype=torch.float32, device="cuda")
        torch.cuda.synchronize()
        for mode, phase in split.schedule(steps, cycle):
            solver.swept_pass(cfg, mode, phase, u.data_ptr(), slots.data_ptr(), sw.native.torch_stream())
        np.testing.assert_array_equal(u.cpu().numpy(), _classic(sw, solver, cfg, ic, steps))
