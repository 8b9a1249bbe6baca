"""The host side of the library without a GPU: ct_api.cu compiled as C++ against tests/native/host_device.cpp, where device
memory is host memory with known blocks and a launch checks that what it was given is there. Allocations are
made to fail on the host; what a later launch is then given must still be live and large enough."""

import ctypes
import os
import pathlib
import subprocess
import sys

import numpy as np
import pytest

ROOT = pathlib.Path(__file__).resolve().parents[1]


@pytest.fixture(scope="module")
def library(tmp_path_factory):
    from cardiotrust_b200 import _lib

    so = tmp_path_factory.mktemp("host_device") / "libhost_device.so"
    _build(so)
    return _lib.load(so)


def _build(so):
    subprocess.check_call(["g++", "-std=c++17", "-O1", "-fPIC", "-shared", "-Wl,-Bsymbolic", "-I/usr/local/cuda/include",
                           "-x", "c++", str(ROOT / "cardiotrust_b200/csrc/ct_api.cu"),
                           str(ROOT / "tests/native/host_device.cpp"), "-o", str(so), "-lpthread", "-ldl"])


class _Host:
    """The compiled library in the place of the real one, and its controls."""

    def __init__(self, lib):
        self.lib = lib
        lib.host_device_live.restype = ctypes.c_size_t

    def fail_from(self, nbytes):
        self.lib.host_device_fail_from(ctypes.c_size_t(nbytes))

    def fail_host_from(self, nbytes):
        self.lib.host_device_fail_host_from(ctypes.c_size_t(nbytes))

    def live(self):
        return int(self.lib.host_device_live())

    def times(self, *ms):
        self.lib.host_device_times((ctypes.c_float * len(ms))(*ms), len(ms))

    def report(self):
        buf = ctypes.create_string_buffer(4096)
        self.lib.host_device_report(buf, len(buf))
        return buf.value.decode()


NEVER = (1 << 63) - 1
#: batches and engines made by a test, closed with the library that they belong to
OPEN = []


def _close_all():
    while OPEN:
        OPEN.pop().close()


@pytest.fixture
def host(library, monkeypatch):
    from cardiotrust_b200 import _lib

    monkeypatch.setattr(_lib, "_LIB", library)
    h = _Host(library)
    h.fail_from(NEVER)
    h.times()
    h.report()
    yield h
    h.fail_from(NEVER)
    _close_all()


@pytest.mark.parametrize("case", ["exchanged", "exchanged_short", "far", "far_short"])
def test_rewired_cases_meet_every_route(host, ctx, case):
    """The scenarios that test_gpu_routes.py runs: tiles followed by progress, by tags and polled directly."""
    import test_gpu_routes as routes

    from cardiotrust_b200 import algorithm as alg

    scn = routes.scenario(*routes.CASES[case])
    scn.measurements = np.zeros((1, scn.control_function.shape[0], scn.num_sensors), np.float32)
    OPEN.append(alg.EpochEngine.from_scenario(ctx, scn, algorithm=alg.Algorithm(freeze_delays=False)))
    far = "far" in routes.CASES[case]
    OPEN[-1].run_epoch(0, grad_mode=alg.GradMode.Reference if far else alg.GradMode.Adjoint, precision=0)
    n = (ctypes.c_int * 6)()
    host.lib.host_device_routes(n)
    progress, tags, polled = n[:3] if far else (min(n[0], n[3]), 3, min(n[2], n[5]))
    assert min(progress, tags, polled) >= 3, list(n)
    assert sum(n[:3]) == 318 and host.report() == ""


@pytest.mark.parametrize("case", ["one_way", "one_way_small", "one_way_ends", "one_way_ends_small"])
def test_one_way_tables_keep_a_short_exchange_ring(host, ctx, case):
    """Tiles that do not read their readers follow a voxel of theirs, so that the ring need not hold the whole beat, in either
    direction; it does once the delays may not fit the staged ring."""
    import test_gpu_routes as routes

    from cardiotrust_b200 import algorithm as alg

    shape, steps, lo, hi, how = routes.CASES[case]
    live = []
    for how in (None, how):
        scn = routes.scenario(shape, steps, lo, hi, how)
        scn.measurements = np.zeros((1, steps, scn.num_sensors), np.float32)
        before = host.live()
        OPEN.append(alg.EpochEngine.from_scenario(ctx, scn, algorithm=alg.Algorithm(freeze_delays=False)))
        OPEN[-1].run_epoch(0, grad_mode=alg.GradMode.Adjoint, precision=0)
        live.append(host.live() - before)
    rows = 16 * int(np.prod(shape))
    assert live[1] - live[0] < 8 * rows
    assert host.report() == ""
    _with_delays(OPEN[-1], 8 + 25)
    OPEN[-1].run_epoch(0, grad_mode=alg.GradMode.Adjoint, precision=0)
    assert host.live() - before - live[1] > (steps - 64) * rows
    assert host.report() == ""


def test_one_way_ring_stays_short_while_the_bounds_are_wide(host, ctx):
    """Delays 8 to 31 fit the staged ring. Epochs that are enqueued ahead widen the host's bounds past it; the device is asked
    before the ring grows to the whole beat."""
    import test_gpu_routes as routes

    from cardiotrust_b200 import algorithm as alg

    shape, steps, _, _, how = routes.CASES["one_way_small"]
    scn = routes.scenario(shape, steps, 8, 31, how)
    scn.measurements = np.zeros((1, steps, scn.num_sensors), np.float32)
    OPEN.append(alg.EpochEngine.from_scenario(ctx, scn, algorithm=alg.Algorithm(freeze_delays=False), num_batch_slots=16))
    before = host.live()
    host.lib.host_device_landed(2)
    for epoch in range(6):
        OPEN[-1].run_epoch(epoch, precision=0, sync=False)
    host.lib.host_device_landed(0)
    assert host.live() == before
    assert host.report() == ""


def _engine(ctx, shape, steps, **kw):
    from cardiotrust_b200 import algorithm as alg
    from cardiotrust_b200 import scenario as sc

    spec = sc.ScenarioSpec(shape=shape, num_steps=steps, num_sensors=3, patho_size=1, patho_origin=(1, 1, 1), seed=2)
    scn = sc.build(spec)
    scn.measurements = np.zeros((1, steps, scn.num_sensors), np.float32)
    OPEN.append(alg.EpochEngine.from_scenario(ctx, scn, num_batch_slots=16, **kw))
    return OPEN[-1]


@pytest.fixture
def ctx(host):
    from cardiotrust_b200 import algorithm as alg

    c = alg.Context(0)
    yield c
    _close_all()
    c.close()


def _batch(ctx, members, **kw):
    from cardiotrust_b200 import algorithm as alg

    engines = [_engine(ctx, *m) for m in members]
    OPEN.append(alg.EpochBatch(ctx, engines, precision=alg.Precision.Fp32, **kw))
    return engines, OPEN[-1]


#: 9, 2 and 2 tiles on 4 CTAs: only the arrangement in one phase needs records for all 13
MEMBERS = [((8, 6, 6), 90), ((4, 4, 4), 70), ((4, 4, 4), 60)]


def test_autotune_without_room_for_one_arrangement(host, ctx):
    """The record of the arrangement in one phase cannot be allocated: the tuner times the others, and the epochs
    that follow use memory that is still there."""
    engines, batch = _batch(ctx, MEMBERS)
    batch.run_epoch()  # a graph that names the first record
    assert host.report() == ""
    before = host.live()
    host.fail_from(1)
    tuned = batch.autotune()
    host.fail_from(NEVER)
    assert tuned["tile_order"] in (0, 1)
    batch.run_epoch()
    assert host.report() == ""
    assert host.live() == before


def test_autotune_gives_back_the_larger_record(host, ctx):
    engines, batch = _batch(ctx, MEMBERS)
    before = host.live()
    host.times(1.0, 2.0, 3.0)  # the first arrangement is the fastest, the last needed the most records
    assert batch.autotune()["tile_order"] == 0
    batch.run_epoch()
    assert host.report() == ""
    assert host.live() == before


def test_autotune_keeps_the_record_of_its_choice(host, ctx):
    engines, batch = _batch(ctx, MEMBERS)
    host.times(3.0, 2.0, 1.0)
    assert batch.autotune()["tile_order"] == 2
    batch.run_epoch()
    assert host.report() == ""


def test_autotune_times_every_arrangement_once(host, ctx):
    """The two epochs that warm up an adjoint batch count for no arrangement, however fast they were."""
    from cardiotrust_b200 import algorithm as alg

    engines, batch = _batch(ctx, MEMBERS, grad_mode=alg.GradMode.Adjoint)
    host.times(1.0, 1.0, 5.0, 4.0, 4.5)
    assert batch.autotune()["tile_order"] == 1
    assert int(batch.batch_indices[0]) == 5
    assert host.report() == ""


def _with_delays(engine, largest):
    d = engine.read("delays")
    d[:] = 8
    d[0, :] = largest
    engine.write("delays", d)


def test_batch_after_an_exchange_ring_that_could_not_grow(host, ctx):
    """A ring that was given back for a longer one, which then did not fit, is made again at its former length: the
    batch's graph must not name the old one, although the lengths agree."""
    from cardiotrust_b200._lib import CtError

    engines, batch = _batch(ctx, [((4, 4, 4), 300), ((4, 4, 4), 200)])
    _with_delays(engines[0], 12)
    batch.run_epoch()
    _with_delays(engines[0], 60)
    host.fail_from(1)
    with pytest.raises(CtError, match="made to fail"):
        engines[0].run_epoch(0, precision=0)
    host.fail_from(NEVER)
    _with_delays(engines[0], 12)
    engines[0].run_epoch(0, precision=0)
    batch.run_epoch()
    assert host.report() == ""


def test_batch_updates_know_the_tables_that_came_later(host, ctx):
    """A reference batch is captured before a member runs its first adjoint epoch by itself: the batch's updates from then on
    cover the delay ranges of that direction."""
    from cardiotrust_b200 import algorithm as alg

    engines, batch = _batch(ctx, MEMBERS)
    for e in engines:
        e.set_freeze(False, False)
        _with_delays(e, 9)  # short enough for the rings to stay as they are
    batch.run_epoch()
    engines[1].run_epoch(0, grad_mode=alg.GradMode.Adjoint, precision=0)
    batch.run_epoch()
    assert host.report() == ""


def test_kernel_follows_the_delays(host, ctx):
    """The recursions' kernel without the direct way runs alone while the delays surely fit the staged ring: exact after a
    write, one step wider on both sides with every update whose read-back has not landed (here: none does). Otherwise
    both are launched, and the device decides."""
    from cardiotrust_b200 import algorithm as alg

    eng = _engine(ctx, (4, 4, 4), 300, algorithm=alg.Algorithm(freeze_delays=False))
    small = _engine(ctx, (4, 4, 4), 200)
    batch = alg.EpochBatch(ctx, [eng, small], precision=alg.Precision.Fp32)
    OPEN.append(batch)
    STAGED, DECIDE = 0, 1
    for largest, routes in ((8 + 24, STAGED), (8 + 25, DECIDE), (20, STAGED)):
        _with_delays(eng, largest)
        eng.simulate()
        assert host.lib.host_device_last_routes() == routes, largest
        batch.run_epoch()  # captured again where the kernel changes
    _with_delays(eng, 20)
    for update in range(10):  # delays 8 to 20: bounds 7 to 21, ..., 1 to 28, where the spread has passed 24
        eng.run_epoch(0, precision=0)
        assert host.lib.host_device_last_routes() == (DECIDE if update > 6 else STAGED), update
    batch.run_epoch()
    assert host.report() == ""


def test_sweep_follows_the_delays(host, ctx):
    """The gradient sweep's kernel without the way for blocks whose delays do not fit its ring runs while they surely do."""
    from cardiotrust_b200 import algorithm as alg

    eng = _engine(ctx, (4, 4, 4), 100, algorithm=alg.Algorithm(freeze_delays=False))
    small = _engine(ctx, (4, 4, 4), 80, algorithm=alg.Algorithm(freeze_delays=False))
    batch = alg.EpochBatch(ctx, [eng, small], precision=alg.Precision.Fp32)
    OPEN.append(batch)
    for largest, wide in ((8 + 16, 0), (8 + 17, 1), (12, 0), (90, 1)):
        _with_delays(eng, largest)
        for mode in (alg.GradMode.Reference, alg.GradMode.Adjoint):
            _with_delays(eng, largest)
            eng.run_epoch(0, grad_mode=mode, precision=0)
            assert host.lib.host_device_last_sweep() == wide, largest
        batch.run_epoch()
    _with_delays(eng, 20)
    for update in range(6):  # delays 8 to 20: bounds 7 to 21, ..., whose spread passes 16 after three updates
        eng.run_epoch(0, precision=0)
        assert host.lib.host_device_last_sweep() == (update > 2), update
    batch.run_epoch()
    assert host.report() == ""


@pytest.mark.parametrize("case, cut", [("far", True), ("far_everywhere", False)])
def test_sweep_blocks_of_scattered_neighbours(host, ctx, case, cut):
    """Blocks end where their halo would not fit, unless that left many of them small: then every block has its eight voxels,
    and the kernel that takes halos of any size runs."""
    import test_gpu_routes as routes

    from cardiotrust_b200 import algorithm as alg

    scn = routes.scenario(*routes.CASES[case])
    scn.measurements = np.zeros((1, scn.control_function.shape[0], scn.num_sensors), np.float32)
    OPEN.append(alg.EpochEngine.from_scenario(ctx, scn, algorithm=alg.Algorithm(freeze_delays=False)))
    OPEN[-1].run_epoch(0, precision=0)
    full = -(-int(np.prod(routes.CASES[case][0])) // 8)
    blocks = host.lib.host_device_sweep_blocks()
    assert full < blocks <= 1.25 * full if cut else blocks == full
    assert host.lib.host_device_last_sweep() == (0 if cut else 1)
    assert host.report() == ""


def test_batch_keeps_its_graph_while_the_bounds_come_and_go(host, ctx):
    """Delays 8 to 31 fit the staged ring. While an update's read-back is under way the bounds are wider and do not; the
    batch captures once for that, not with every change."""
    from cardiotrust_b200 import algorithm as alg

    engines, batch = _batch(ctx, MEMBERS[1:])
    for e in engines:
        e.set_freeze(False, False)
        _with_delays(e, 8 + 23)
    batch.run_epoch()
    host.lib.host_device_captures()
    for epoch in range(14):
        host.lib.host_device_landed(epoch // 2 % 2)
        batch.run_epoch()
    host.lib.host_device_landed(0)
    assert host.lib.host_device_captures() == 1
    assert host.report() == ""


def test_delays_above_the_roll_limit_keep_their_ring(host, ctx):
    """An update moves no delay past 1,000, but leaves a larger one that was written where it is: the ring that is
    sized afterwards holds the rows that it reads."""
    from cardiotrust_b200 import algorithm as alg

    eng = _engine(ctx, (4, 4, 4), 4200, algorithm=alg.Algorithm(freeze_delays=False))
    _with_delays(eng, 1500)
    eng.run_epoch_plain(0)  # an update, before any recursion has asked for its ring
    eng.run_epoch(0, precision=0)
    assert host.report() == ""


def test_adjoint_tables_of_a_lattice(host, ctx):
    """The adjoint's direction shares the forward's halo tables on a lattice: less memory than tables of its own, and a
    refused allocation leaves nothing behind."""
    from cardiotrust_b200 import algorithm as alg
    from cardiotrust_b200._lib import CtError

    eng = _engine(ctx, (8, 6, 6), 10)
    before = host.live()
    host.fail_from(4 * 10 * 3 * 288)  # the gradient of the states
    with pytest.raises(CtError, match="made to fail"):
        eng.run_epoch(0, grad_mode=alg.GradMode.Adjoint, precision=0)
    host.fail_from(NEVER)
    assert host.live() == before
    eng.run_epoch(0, grad_mode=alg.GradMode.Adjoint, precision=0)
    own = 9 * 192 * (4 + 2)  # halos and their slots
    assert host.live() - before - 4 * 10 * 3 * 288 < 288 * 26 * (4 + 2) + own
    eng.run_epoch(0, grad_mode=alg.GradMode.Reference, precision=0)
    OPEN.pop().close()
    assert host.live() == 0
    assert host.report() == ""


#: no thread can be started, then each size of host allocation fails: a status each time, never an abort
CHILD = """
import sys
sys.path[:0] = [{root!r}, {tests!r}]
import pathlib
import test_host_device as t
from cardiotrust_b200 import _lib, algorithm as alg
_lib._LIB = _lib.load(pathlib.Path({so!r}))
host = t._Host(_lib._LIB)
ctx = alg.Context(0)
host.lib.host_device_no_threads(1)
t._engine(ctx, (4, 4, 4), 50)
t._close_all()
print("without threads")
host.lib.host_device_no_threads(0)
before, refused = host.live(), 0
for bits in range(4, 24):
    host.fail_host_from(1 << bits)
    try:
        engines, batch = t._batch(ctx, t.MEMBERS, grad_mode=alg.GradMode.Adjoint)
        batch.run_epoch()
        batch.autotune()
        engines[0].run_epoch(0, precision=0)
    except _lib.CtError as e:
        assert e.status == _lib.CT_ERR_OUT_OF_MEMORY, e
        refused += 1
    host.fail_host_from(t.NEVER)
    t._close_all()
    assert host.live() == before and host.report() == "", (bits, host.live(), before)
print("refused", refused)
"""


def test_host_failures_are_reported(tmp_path):
    so = tmp_path / "libhost_device.so"
    _build(so)
    code = CHILD.format(root=str(ROOT), tests=str(ROOT / "tests"), so=str(so))
    done = subprocess.run([sys.executable, "-c", code], env=dict(os.environ, LD_PRELOAD=str(so)), capture_output=True,
                          text=True, timeout=300)
    assert done.returncode == 0, done.stdout + done.stderr
    assert "without threads" in done.stdout and int(done.stdout.split("refused")[1]) >= 8
