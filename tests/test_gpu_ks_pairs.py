"""FP32 KS swept passes with two tiles per block (csrc/swept_pair.cuh) against the
oracle, bit for bit: the smallest domains that take that path, odd tile counts
(the last block's tile in both halves), the wrapping phase-1 tile paired and
alone, one and two position groups per thread, tile widths that are no power
of two, both forms of the right-hand side, and ensembles whose pairs straddle
domains."""
import importlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

KS, SWEPT, TIME_STEPS = 1, 1, 1
ens = importlib.import_module("1dsweptcuda_gb300.ensemble")


def _ic(n, seed):
    rng = np.random.default_rng(seed)
    x = np.arange(n)
    return (np.cos(2 * np.pi * 5 * x / n) + 0.1 * rng.standard_normal(n)).astype(np.float32)


def _sms():
    torch = pytest.importorskip("torch")
    return torch.cuda.get_device_properties(0).multi_processor_count


@pytest.mark.parametrize("dx, dt", [(0.5, 0.005), (0.3, 5e-4)])
@pytest.mark.parametrize("tpb, per_sm, extra", [(128, 8, 1), (128, 8, 2), (160, 1, 1), (192, 1, 1), (256, 1, 1), (256, 1, 2),
                                                (512, 1, 2), (640, 1, 3), (1024, 1, 1), (768, 16, 0), (1024, 16, 1)])
def test_pairs_equal_the_oracle(sw, solver, oracle, tpb, per_sm, extra, dx, dt):
    nx = tpb * (per_sm * _sms() + extra)
    ic = _ic(nx, tpb + extra)
    c = oracle.ks_consts(4, nx, dt, dx=dx)
    cycle = tpb // 8
    for steps in (cycle, 2 * cycle + 1, 3 * cycle):
        cfg = sw.make_config(KS, 4, alg=SWEPT, nx=nx, tpb=tpb, dt=dt, dx=dx, time_mode=TIME_STEPS, n_steps=steps)
        got, _, _ = solver.run(cfg, ic)
        np.testing.assert_array_equal(got, oracle.classic(c, ic, steps), err_msg="steps %d" % steps)


@pytest.mark.parametrize("dx, dt", [(0.5, 0.005), (0.3, 5e-4)])
def test_pairs_across_domains(sw, solver, oracle, dx, dt):
    tpb = 256
    nx = tpb * np.array([1, 64, 3, 101, 2, 1, 97], dtype=np.int64)  # 269 tiles: odd counts, single tiles
    ic = np.concatenate([_ic(int(n), i) for i, n in enumerate(nx)])
    steps = 3 * (tpb // 8) + 2
    cfg = sw.make_config(KS, 4, alg=SWEPT, tpb=tpb, dt=dt, dx=dx, time_mode=TIME_STEPS, n_steps=steps)
    got, _ = solver.run_batch(cfg, nx, ic)
    want = ens.concat([oracle.classic(oracle.ks_consts(4, int(n), dt, dx=dx), part, steps)
                       for part, n in zip(ens.split(ic, nx, 1), nx)])
    np.testing.assert_array_equal(got, want)


def test_pairs_of_extreme_values(sw, solver, oracle):
    """Overflowing squares, infinities' and NaNs' spread, zeros of both signs and subnormals."""
    tpb, dt = 256, 0.005
    nx = tpb * (_sms() + 1)
    ic = _ic(nx, 9)
    ic[1000:1004] = [0.0, -0.0, 1e-42, -1e-42]
    ic[30000] = 3e19
    c = oracle.ks_consts(4, nx, dt)
    cfg = sw.make_config(KS, 4, alg=SWEPT, nx=nx, tpb=tpb, dt=dt, time_mode=TIME_STEPS, n_steps=65)
    got, want = solver.run(cfg, ic)[0], oracle.classic(c, ic, 65)
    assert np.isnan(want).any() and not np.isnan(want).all()
    np.testing.assert_array_equal(got, want)
