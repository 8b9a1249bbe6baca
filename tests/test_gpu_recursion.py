"""The recursions through time and the gradient sweep, where their routes part: hand-overs of one and two steps
(smallest delay 1, 2 and 3), delays that wrap the shared history ring or do not fit it, partly filled and
single tiles, more tiles than CTAs, neighbour tables that are not symmetric, and beats shorter than the delays.

States are bit-identical to the f32 oracle and reference-mode gradients to its CPU loop up to the rounding
of the mapped residuals (the products' bar, 1e-3); adjoint gradients are held to 1e-3 of the f64 oracle, the
stated gradient tolerance."""

import dataclasses

import numpy as np
import pytest

from conftest import oracle_forward, rel_err

pytestmark = pytest.mark.gpu

TOL_GRAD = 1e-3

#: name -> (grid, steps, smallest and largest delay, share of one-way connections that are cut)
CASES = {
    "delay_1": ((4, 4, 4), 61, 1, 1, 0.0),
    "delays_1_to_2": ((5, 3, 7), 64, 1, 2, 0.0),
    "delays_2_to_5": ((4, 5, 9), 75, 2, 5, 0.0),
    "delays_3_to_9_odd_end": ((7, 5, 6), 77, 3, 9, 0.0),
    "ring_full": ((6, 5, 5), 120, 5, 28, 0.0),
    "ring_overflow": ((6, 5, 5), 120, 5, 60, 0.0),
    "beat_below_delays": ((4, 4, 5), 6, 7, 40, 0.0),
    "one_step": ((3, 3, 3), 1, 1, 4, 0.0),
    "two_steps": ((3, 3, 3), 2, 1, 1, 0.0),
    "one_way": ((6, 6, 5), 90, 4, 9, 0.3),
    "one_way_short_delays": ((5, 5, 5), 70, 1, 3, 0.5),
    "scattered": ((6, 6, 5), 70, 3, 8, 0.2),
    "several_tiles_per_cta": ((22, 21, 22), 50, 8, 14, 0.0),
    "several_tiles_delays_1_to_3": ((22, 21, 22), 37, 1, 3, 0.0),
    "several_tiles_ring_overflow": ((22, 21, 22), 45, 2, 40, 0.1),
}


@pytest.fixture(scope="module")
def alg():
    from cardiotrust_b200 import algorithm

    return algorithm


@pytest.fixture(scope="module")
def ctx(alg):
    c = alg.Context(0)
    yield c
    c.close()


def _scenario(oracle_mod, case):
    from cardiotrust_b200 import scenario as sc

    shape, steps, lo, hi, cut = CASES[case]
    spec = sc.ScenarioSpec(shape=shape, num_steps=steps, num_sensors=5, patho_size=2, patho_origin=(1, 1, 1), pulse_onset=0,
                           pulse_sigma_samples=2.0, seed=11)
    scn = sc.build(spec)
    rng = np.random.default_rng(len(case))

    def vary(p):
        connected = p.output_state_indices[::3, ::3] >= 0  # [V, 26]
        keep = connected & (draw >= cut)
        to = p.output_state_indices
        if case == "scattered":  # neighbours anywhere: halos of many voxels, cut blocks
            to = np.repeat(3 * np.repeat(where, 3, axis=0), 3, axis=1) + np.tile(np.arange(3), 26)
        osi = np.where(np.repeat(np.repeat(keep, 3, axis=0), 3, axis=1), to, -1).astype(np.int32)
        # gains on every connection, damped so that 26 of them with short delays do not grow
        gains = np.where(osi >= 0, gain, 0.0).astype(np.float32)
        return dataclasses.replace(p, output_state_indices=osi, delays=np.where(keep, delays, p.delays).astype(np.int32),
                                   gains=gains)

    V = scn.model.coefs.shape[0]
    draw = rng.random((V, 26))
    where = np.argsort(np.random.default_rng(1).random((V, V)), axis=1)[:, :26] if case == "scattered" else None
    delays = rng.integers(lo, hi + 1, size=(V, 26))
    delays[0, :], delays[-1, :] = lo, hi  # both ends occur
    gain = rng.normal(0.0, 0.06, size=(3 * V, 78))
    scn = dataclasses.replace(scn, model=vary(scn.model), truth=vary(scn.truth))
    scn.truth = dataclasses.replace(scn.truth, gains=(scn.truth.gains * np.float32(0.9)).astype(np.float32))
    return sc.attach_measurements(scn, oracle_forward(oracle_mod))


@pytest.mark.parametrize("case", sorted(CASES))
def test_recursions_and_sweep(alg, ctx, oracle_mod, case):
    scn = _scenario(oracle_mod, case)
    a = alg.Algorithm(learning_rate=0.0, freeze_delays=False, maximum_regularization_threshold=0.5)
    oa = oracle_mod.algo(learning_rate=0.0, freeze_delays=0, maximum_regularization_threshold=0.5)
    eng = alg.EpochEngine.from_scenario(ctx, scn, algorithm=a)

    eng.run_epoch(0)
    o32 = oracle_mod.from_scenario(scn)
    o32.run_epoch(oa)
    np.testing.assert_array_equal(eng.read("system_states").view(np.uint32), o32.system_states.view(np.uint32))
    for name, want in (("ap_outputs_now", o32.ap_outputs_now), ("ap_outputs_last", o32.ap_outputs_last)):
        np.testing.assert_array_equal(eng.read(name), want)
    assert rel_err(eng.read("grad_gains"), o32.d_gains) < TOL_GRAD
    assert rel_err(eng.read("grad_coefs"), o32.d_coefs) < TOL_GRAD
    assert rel_err(eng.read("loss_maximum_regularization"), o32.loss_maximum_regularization) < 1e-4

    if case == "scattered":  # the adjoint wants a lattice
        eng.close()
        return
    eng.run_epoch(0, grad_mode=alg.GradMode.Adjoint)
    o64 = oracle_mod.from_scenario(scn, dtype=np.float64)
    o64.run_epoch(oa, adjoint=True)
    assert rel_err(eng.read("grad_gains"), o64.d_gains) < TOL_GRAD
    assert rel_err(eng.read("grad_coefs"), o64.d_coefs) < TOL_GRAD
    eng.close()


@pytest.mark.parametrize("case", ["delays_3_to_9_odd_end", "scattered", "several_tiles_per_cta", "several_tiles_ring_overflow"])
@pytest.mark.parametrize("kw", [{}, {"ap_derivative": 0}, {"freeze_gains": True}, {"freeze_delays": True}],
                         ids=["textbook", "simple", "coefs_only", "gains_only"])
def test_sweep_bits(alg, ctx, oracle_mod, case, kw):
    """With and without the shared history, whole and cut blocks: bit for bit the CPU loop, given the mapped residuals."""
    scn = _scenario(oracle_mod, case)
    shared = dict(learning_rate=0.0, maximum_regularization_threshold=0.5, difference_regularization_strength=1e-3)
    a = alg.Algorithm(**shared, **{"freeze_delays": False, **kw,
                                   "ap_derivative": alg.APDerivative(kw.get("ap_derivative", 1))})
    oa = oracle_mod.algo(**shared, **{"freeze_delays": 0, **{k: int(v) for k, v in kw.items()}})
    eng = alg.EpochEngine.from_scenario(ctx, scn, algorithm=a)
    eng.run_epoch(0)
    o = oracle_mod.from_scenario(scn)
    o.mapped_residuals_override = np.ascontiguousarray(eng.read("mapped_residuals_history")[None])
    o.run_epoch(oa)
    for name, want in (("grad_gains", o.d_gains), ("grad_coefs", o.d_coefs), ("coefs_fir", o.coefs_fir),
                       ("coefs_iir", o.coefs_iir)):
        if (name == "grad_gains" and a.freeze_gains) or (name != "grad_gains" and a.freeze_delays):
            continue
        np.testing.assert_array_equal(eng.read(name).view(np.uint32), want.view(np.uint32), err_msg=name)
    eng.close()


def test_batch_phases_match_single_runs(alg, ctx, oracle_mod):
    """A batch whose members differ in tiles per CTA, delays and beat lengths, in every arrangement of its tiles."""
    names = ["several_tiles_per_cta", "delays_2_to_5", "ring_overflow", "one_way", "several_tiles_delays_1_to_3"]
    scns = [_scenario(oracle_mod, n) for n in names]
    a = alg.Algorithm(learning_rate=0.0, freeze_delays=False)
    for mode in (alg.GradMode.Reference, alg.GradMode.Adjoint):
        want = []
        for s in scns:
            e = alg.EpochEngine.from_scenario(ctx, s, algorithm=a, num_batch_slots=8)
            e.run_epoch(0, grad_mode=mode)
            want.append((e.read("system_states"), e.read("grad_gains"), e.read("grad_coefs")))
            e.close()
        engines = [alg.EpochEngine.from_scenario(ctx, s, algorithm=a, num_batch_slots=8) for s in scns]
        batch = alg.EpochBatch(ctx, engines, grad_mode=mode)
        batch.autotune()  # runs an epoch in every arrangement
        batch.run_epoch()
        for e, w in zip(engines, want):
            for name, ref in zip(("system_states", "grad_gains", "grad_coefs"), w):
                np.testing.assert_array_equal(e.read(name).view(np.uint32), ref.view(np.uint32))
        batch.close()
        for e in engines:
            e.close()
