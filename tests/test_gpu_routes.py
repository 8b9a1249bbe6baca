"""Tiles on different routes of the recursion kernel in one launch: followed by the progress of the tiles around, by the
tags of their rows, and polled directly, alone on a CTA or several in turn; pairs of steps across the visits of a
CTA; layers of tissue with other delays; tiles that are read by tiles that they do not read; a batch's small members in the places that a large one leaves free.

States are bit-identical to the f32 oracle. Gradients lie within 1e-5 of the oracle (adjoint: f64; reference: the f32 loop),
ten times the rounding of sums of this length in f32."""

import dataclasses

import numpy as np
import pytest

from conftest import oracle_forward, rel_err

TOL = 1e-5
SHAPE = (22, 21, 22)  # 318 tiles, more than the CTAs of a device of 148 SMs


def rewired(p, rng, how, shape=SHAPE):
    """Voxels of the last layer that a walk from voxel 0 reaches get other neighbours, most of a tile's voxels in some places, a
    few in others. "exchanged": each other's, so that along each offset still no two voxels reach the same one.
    "far": anywhere in the grid ("far_everywhere": those of every voxel)."""
    V = p.coefs.shape[0]
    nbr = np.where(p.output_state_indices[::3, ::3] >= 0, p.output_state_indices[::3, ::3] // 3, -1)
    x, y, z = np.unravel_index(np.arange(V), shape)
    last = (x == shape[0] - 1) | (z == shape[2] - 1)
    place = (y // 4 + z // 4 + x // 4) % 3
    w = np.nonzero(last & (rng.random(V) < np.array([0.9, 0.2, 0.0])[place]))[0]
    if how == "far_everywhere":
        w = np.arange(V)
    if how.startswith("far"):
        nbr[w] = np.argsort(rng.random((w.size, V)), axis=1)[:, :26]
    else:
        for n in range(26):
            nbr[w, n] = nbr[rng.permutation(w), n]
    to = np.repeat(3 * np.repeat(nbr, 3, axis=0), 3, axis=1) + np.tile(np.arange(3), 26)
    return np.where(np.repeat(np.repeat(nbr, 3, axis=0), 3, axis=1) >= 0, to, -1).astype(np.int32)


def one_way(p, shape, ends):
    """Voxels from the third brick on read none before it, or, as ends of the activation's way, none at all."""
    osi = p.output_state_indices.copy()
    x = np.unravel_index(np.arange(osi.shape[0] // 3), shape)[0]
    behind = np.repeat(x >= 8, 3)
    osi[behind[:, None] & ((np.repeat(x, 3)[np.maximum(osi, 0)] < 8) | ends)] = -1
    return osi


def scenario(shape, steps, lo, hi, how=None, beats=1):
    from cardiotrust_b200 import scenario as sc

    spec = sc.ScenarioSpec(shape=shape, num_steps=steps, num_beats=beats, num_sensors=5, patho_size=2, patho_origin=(1, 1, 1),
                           pulse_onset=0, pulse_sigma_samples=2.0, seed=13)
    scn = sc.build(spec)
    rng = np.random.default_rng(steps)
    osi = rewired(scn.model, rng, how, shape) if how in ("exchanged", "far", "far_everywhere") else scn.model.output_state_indices
    if how in ("one_way", "ends"):
        osi = one_way(scn.model, shape, how == "ends")
    if how == "alone":
        osi = np.full_like(scn.model.output_state_indices, -1)
    connected = osi[::3, ::3] >= 0
    drawn = rng.integers(lo, hi + 1, size=connected.shape)
    if how == "layers":  # a slow layer and a fast one, as tissues with other velocities make them
        z = np.arange(connected.shape[0]) % shape[2]
        drawn[z // 4 == 1] = rng.integers(60, 121, size=drawn.shape)[z // 4 == 1]
        drawn[z // 4 == 3] = rng.integers(1, 4, size=drawn.shape)[z // 4 == 3]
    drawn[0, :], drawn[-1, :] = lo, hi  # both ends occur
    delays = np.where(connected, drawn, scn.model.delays).astype(np.int32)
    gain = rng.normal(0.0, 0.06, size=osi.shape)  # damped, so that 26 connections do not grow

    def vary(p, scale):
        return dataclasses.replace(p, output_state_indices=osi, delays=delays,
                                   gains=np.where(osi >= 0, scale * gain, 0.0).astype(np.float32))

    return dataclasses.replace(scn, model=vary(scn.model, 1.0), truth=vary(scn.truth, 0.9))


#: name -> grid, steps, smallest and largest delay, rewired how
CASES = {
    "exchanged": (SHAPE, 47, 6, 11, "exchanged"),
    "exchanged_short": (SHAPE, 33, 1, 4, "exchanged"),
    "far": (SHAPE, 47, 6, 11, "far"),
    "far_short": (SHAPE, 33, 2, 4, "far"),
    "far_everywhere": ((13, 16, 14), 60, 4, 9, "far_everywhere"),
    "far_everywhere_small": ((7, 6, 5), 90, 4, 9, "far_everywhere"),
    "layers": (SHAPE, 150, 6, 12, "layers"),
    "layers_small": ((7, 6, 19), 260, 6, 12, "layers"),
    "alone": (SHAPE, 150, 4, 9, "alone"),
    "one_way": (SHAPE, 150, 4, 9, "one_way"),
    "one_way_small": ((13, 6, 7), 300, 4, 9, "one_way"),
    "one_way_ends": (SHAPE, 150, 4, 9, "ends"),
    "one_way_ends_small": ((13, 6, 7), 300, 4, 9, "ends"),
    "smallest_3": (SHAPE, 41, 3, 9),
    "smallest_7": (SHAPE, 50, 7, 12),
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


@pytest.mark.gpu
@pytest.mark.parametrize("case", sorted(CASES))
def test_routes(alg, ctx, oracle_mod, case):
    from cardiotrust_b200 import scenario as sc

    scn = sc.attach_measurements(scenario(*CASES[case]), oracle_forward(oracle_mod))
    kw = dict(learning_rate=0.0, maximum_regularization_threshold=0.5)
    eng = alg.EpochEngine.from_scenario(ctx, scn, algorithm=alg.Algorithm(freeze_delays=False, **kw))
    oa = oracle_mod.algo(freeze_delays=0, **kw)

    eng.run_epoch(0, precision=alg.Precision.Fp32)
    o32 = oracle_mod.from_scenario(scn)
    o32.mapped_residuals_override = np.ascontiguousarray(eng.read("mapped_residuals_history")[None])
    o32.run_epoch(oa)
    np.testing.assert_array_equal(eng.read("system_states").view(np.uint32), o32.system_states.view(np.uint32))
    np.testing.assert_array_equal(eng.read("grad_gains").view(np.uint32), o32.d_gains.view(np.uint32))
    np.testing.assert_array_equal(eng.read("grad_coefs").view(np.uint32), o32.d_coefs.view(np.uint32))

    if "far" in case:  # two voxels reach the same one: refused
        with pytest.raises(alg.CtError, match="not a lattice"):
            eng.run_epoch(0, grad_mode=alg.GradMode.Adjoint, precision=alg.Precision.Fp32)
        eng.close()
        return
    eng.run_epoch(0, grad_mode=alg.GradMode.Adjoint, precision=alg.Precision.Fp32)
    o64 = oracle_mod.from_scenario(scn, dtype=np.float64)
    o64.run_epoch(oa, adjoint=True)
    assert rel_err(eng.read("grad_gains"), o64.d_gains) < TOL
    assert rel_err(eng.read("grad_coefs"), o64.d_coefs) < TOL
    eng.close()


#: a large member, and small ones with shorter beats, which fill the places that it leaves free
MEMBERS = [(SHAPE, 60, 8, 14), ((5, 4, 6), 40, 2, 5), ((6, 5, 5), 50, 3, 40), ((4, 4, 4), 20, 1, 2)]


@pytest.mark.gpu
@pytest.mark.parametrize("mode", [0, 1], ids=["reference", "adjoint"])
def test_batch_fills_free_places(alg, ctx, oracle_mod, mode):
    """The default arrangement, the last one that the tuner tries (it leaves its results) and the one that it chooses."""
    from cardiotrust_b200 import scenario as sc

    mode = alg.GradMode(mode)
    names = ("system_states", "grad_gains", "grad_coefs", "loss")
    a = alg.Algorithm(learning_rate=0.0, freeze_delays=False)
    scns = [sc.attach_measurements(scenario(*m, beats=1 + i % 2), oracle_forward(oracle_mod)) for i, m in enumerate(MEMBERS)]
    want = []
    for s in scns:
        e = alg.EpochEngine.from_scenario(ctx, s, algorithm=a)
        e.run_epoch(0, beat_order=np.arange(s.measurements.shape[0], dtype=np.int32), grad_mode=mode)
        want.append([e.read(n) for n in names])
        e.close()
    engines = [alg.EpochEngine.from_scenario(ctx, s, algorithm=a, num_batch_slots=8) for s in scns]
    batch = alg.EpochBatch(ctx, engines, grad_mode=mode)

    def compare(what):
        for e, w in zip(engines, want):
            for n, ref in zip(names, w):
                np.testing.assert_array_equal(e.read(n).view(np.uint32), ref.view(np.uint32), err_msg=f"{what}: {n}")

    batch.run_epoch()
    compare("default")
    batch.autotune()
    compare("one phase")
    batch.run_epoch()
    compare("chosen")
    batch.close()
    for e in engines:
        e.close()
