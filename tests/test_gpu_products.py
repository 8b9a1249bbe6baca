"""The FP32 products H x and H^T r where their blocks part: one and two column widths, remainders of rows, columns and
inner length, rows that start on 16 bytes and rows that do not, one and several splits. Every value lies within
the bound of an FP32 sum of its terms in any order, (number of terms + splits) 2^-24 sum |a b|, of the FP64 product."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EPS = 2.0 ** -24


def _within(got, a, b, terms):
    a, b = a.astype(np.float64), b.astype(np.float64)
    bound = 1.01 * terms * EPS * (np.abs(a) @ np.abs(b))
    assert (np.abs(got.astype(np.float64) - a @ b) <= bound).all()


@pytest.mark.parametrize("T,S,M", [(1, 3, 1), (127, 135, 63), (128, 256, 64), (129, 260, 65), (130, 768, 128), (257, 1023, 129),
                                   (300, 1536, 111), (64, 2052, 192), (40, 4100, 256)])
def test_predicted_measurements(T, S, M):
    import torch

    from cardiotrust_b200 import _lib

    rng = np.random.default_rng(T + S + M)
    x, h = (rng.standard_normal(n).astype(np.float32) for n in ((T, S), (M, S)))
    X, H = torch.from_numpy(x).cuda(), torch.from_numpy(h).cuda()
    Y = torch.full((T, M), float("nan"), device="cuda")
    _lib.check(_lib.lib().ct_predict_measurements_noalloc(X.data_ptr(), H.data_ptr(), None, Y.data_ptr(), None, T, S, M, None))
    torch.cuda.synchronize()
    _within(Y.cpu().numpy(), x, h.T, S + 64)


@pytest.mark.parametrize("shape,steps,sensors", [((5, 3, 3), 129, 1), ((5, 3, 3), 200, 21), ((4, 4, 4), 128, 4), ((5, 5, 5), 131, 48),
                                                 ((8, 7, 6), 127, 43)])
def test_mapped_residuals(shape, steps, sensors):
    from cardiotrust_b200 import algorithm as alg
    from cardiotrust_b200 import scenario as sc

    spec = sc.ScenarioSpec(shape=shape, num_steps=steps, num_sensors=sensors, patho_size=1, patho_origin=(1, 1, 1),
                           pulse_onset=1, pulse_sigma_samples=4.0, seed=5)
    scn = sc.build(spec)
    rng = np.random.default_rng(sensors)
    scn.measurements = rng.standard_normal((1, steps, scn.num_sensors)).astype(np.float32)
    ctx = alg.Context(0)
    eng = alg.EpochEngine.from_scenario(ctx, scn, algorithm=alg.Algorithm(learning_rate=0.0, freeze_delays=False))
    eng.run_epoch(0, precision=alg.Precision.Fp32)
    r = eng.read("measurements")[0] - scn.measurements[0]
    _within(eng.read("mapped_residuals_history"), r, scn.measurement_matrix[0], scn.num_sensors)
    eng.close()
    ctx.close()
