"""The host layer's decisions (capi.cpp) against a CUDA runtime that only keeps books (fake_cuda.cpp): what a call
does when a capture, an allocation or a launch fails, which memory is held when, and what the autotuners pick
when the costs are known."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from mrlbm_2d_b200 import api
from mrlbm_2d_b200.config import cylinder_case

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "mrlbm_2d_b200", "csrc")
CUDA_INC = "/usr/local/cuda/include"
STEP, PAIR, BATCH = 0, 1, 2

fake_args = dict(fake_limit=[ctypes.c_int64], fake_pair_us=[ctypes.c_double], fake_graph_factor=[ctypes.c_double], fake_step_us=[ctypes.c_int, ctypes.c_double],
                 fake_fail=[ctypes.c_char_p, ctypes.c_int], fake_fail_after=[ctypes.c_char_p, ctypes.c_int, ctypes.c_int])

pytestmark = pytest.mark.skipif(not os.path.isdir(CUDA_INC), reason="CUDA headers not installed")


@pytest.fixture(scope="module")
def library(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("fake") / "libfake.so")
    srcs = [os.path.join(CSRC, f) for f in ("capi.cpp", "geometry.cpp", "statistics.cpp")]
    subprocess.run(["g++", "-std=c++17", "-O1", "-fPIC", "-shared", "-Wl,-Bsymbolic", "-I", CSRC, "-I", os.path.join(ROOT, "include"), "-I", CUDA_INC,
                    *srcs, os.path.join(ROOT, "tests", "fake_cuda.cpp"), "-o", out], check=True)
    L = api.load_library(out)
    for f in ("fake_used", "fake_peak", "fake_done", "fake_captures", "fake_graphs", "fake_dangling"):
        getattr(L, f).restype = ctypes.c_int64
    for f, a in fake_args.items():
        getattr(L, f).argtypes = a
    return L


@pytest.fixture
def fake(library, monkeypatch):
    monkeypatch.setattr(api, "_lib", library)
    monkeypatch.delenv("MRLBM_PAIRS", raising=False)
    library.fake_reset()
    yield library
    assert library.fake_dangling() == 0


def small():
    return cylinder_case(120, 48, 12, 30.0, 24.5, 100.0, 0.05)


def large():
    """Above the size from which FP64 steps are taken in pairs."""
    return cylinder_case(1400, 520, 40, 300.0, 260.5, 100.0, 0.05)


def tuned_pairs(fake):
    """Costs at which every autotuner takes pairs."""
    fake.fake_pair_us(0.5)


@pytest.mark.parametrize("prec", [64, 32])
@pytest.mark.parametrize("call", ["cudaMalloc", "cudaStreamBeginCapture", "launch", "cudaStreamEndCapture", "cudaGraphInstantiate",
                                  "cudaMemcpyAsync", "cudaGraphLaunch"])
def test_a_replay_that_cannot_be_made_is_launched_step_by_step(fake, prec, call):
    s = api.Simulation(small(), precision=prec)
    fake.fake_fail(call.encode(), 1)                         # the first call of its kind is the replay's
    s.step(2600)
    assert s.iter == 2601 and fake.fake_done(STEP) == 2600
    captures = fake.fake_captures()
    s.step(2600)                                             # not tried again for every run
    assert fake.fake_captures() == captures and fake.fake_done(STEP) == 5200
    s.close()


LATER = {"macro": lambda s: s.step(5, macro=True), "field window": lambda s: s.field_stats_window(2, 100), "state": lambda s: s.get_state(),
         "body force": lambda s: s.set_body_force(np.zeros((2, s.nx, s.ny))), "inlet profile": lambda s: s.set_inlet_profile(np.zeros(s.ny)),
         "surface": lambda s: s.surface_enable(), "gradient": lambda s: s.adjoint_drag(20, 5, 6), "autotune": lambda s: s.autotune(4)}


@pytest.mark.parametrize("what", sorted(LATER))
def test_the_band_of_the_pairs_goes_back_when_memory_is_short(fake, monkeypatch, what):
    """What fits beside a handle of single steps fits beside one that steps in pairs."""
    cfg = large()
    monkeypatch.setenv("MRLBM_PAIRS", "0")
    s = api.Simulation(cfg)
    single = fake.fake_used()
    fake.fake_mark()
    LATER[what](s)
    need = fake.fake_peak()
    s.close()
    monkeypatch.delenv("MRLBM_PAIRS")
    s = api.Simulation(cfg)
    assert fake.fake_used() == single + s.info.state_bytes // 2          # pairs, with their third level
    s.step(4)
    assert fake.fake_done(PAIR) == 2
    fake.fake_limit(max(need, fake.fake_used()))
    LATER[what](s)
    pairs = fake.fake_done(PAIR)
    s.step(4)
    assert s.status() == 0
    if need > single + s.info.state_bytes // 2:
        assert fake.fake_done(PAIR) == pairs                             # single steps since
    s.close()


def test_pairs_take_at_most_a_quarter_of_the_free_memory(fake):
    cfg = large()
    s = api.Simulation(cfg)
    level, used = s.info.state_bytes // 2, fake.fake_used()
    s.close()
    for room, pairs in ((4 * level + 1000, 2), (4 * level - 1000, 0)):
        fake.fake_reset()
        fake.fake_limit(used - level + room)
        s = api.Simulation(cfg)
        s.step(4)
        assert fake.fake_done(PAIR) == pairs
        s.close()


@pytest.mark.parametrize("forced", [False, True])
def test_a_batch_is_created_in_the_memory_of_single_steps(fake, monkeypatch, forced):
    cfgs = [large()] * 3
    monkeypatch.setenv("MRLBM_PAIRS", "0")
    fake.fake_mark()
    b = api.Batch(cfgs, precision=64)
    single = fake.fake_peak()
    b.close()
    if forced:
        monkeypatch.setenv("MRLBM_PAIRS", "1")
        fake.fake_limit(single)
    else:
        monkeypatch.delenv("MRLBM_PAIRS")
    fake.fake_mark()
    b = api.Batch(cfgs, precision=64)
    assert fake.fake_peak() == single
    fake.fake_limit(1 << 62)
    b.step(10)
    assert b.status() == 0
    b.close()


def test_a_batch_in_pairs_gives_its_bands_back(fake):
    cfgs = [large()] * 3
    b = api.Batch(cfgs, precision=64)
    used = fake.fake_used()
    tuned_pairs(fake)
    b.autotune(8)
    assert fake.fake_used() > used + 3 * (b.cases[0].info.state_bytes // 2)
    b.step(16)
    pairs = fake.fake_done(PAIR)
    assert pairs > 0
    fake.fake_limit(fake.fake_used() + 1000)
    b.step(16, macro=True)                                               # three macroscopic buffers
    b.step(16)
    assert b.status() == 0
    b.close()


def test_a_schedule_set_by_hand_has_no_pairs_but_the_autotuners_has(fake):
    b = api.Batch([large()] * 2, precision=64)
    single = fake.fake_used()
    tuned_pairs(fake)
    tuned, _ = b.autotune(8)
    paired = fake.fake_used()
    b.set_schedule(3, api.BATCH_STREAMS, 8)
    assert fake.fake_used() == paired - 2 * (b.cases[0].info.state_bytes // 2)    # the bands are back
    pairs = fake.fake_done(PAIR)
    b.step(16)
    assert fake.fake_done(PAIR) == pairs
    b.set_schedule(*tuned)
    assert b.schedule == tuned and fake.fake_used() >= single + b.cases[0].info.state_bytes
    b.step(16)
    assert fake.fake_done(PAIR) == pairs + 16                                     # 8 pairs of each case
    b.close()


@pytest.mark.parametrize("call", ["pair", "cudaGraphLaunch"])
def test_batch_autotune_without_pairs_when_their_trial_fails(fake, call):
    b = api.Batch([large()] * 2, precision=64)
    tuned_pairs(fake)
    used = fake.fake_used()
    if call == "cudaGraphLaunch":                            # the paired trial's: after those of the shapes
        fake.fake_reset()
        tuned_pairs(fake)
        b.autotune(8)
        n = fake.fake_graphs()
        b.close()
        fake.fake_reset()
        tuned_pairs(fake)
        b = api.Batch([large()] * 2, precision=64)
        used = fake.fake_used()
        fake.fake_fail_after(call.encode(), n - 4, 1)
    else:
        fake.fake_fail(b"pair", 1)
    b.autotune(8)
    level = b.cases[0].info.state_bytes // 2
    assert fake.fake_used() < used + level                   # no bands
    b.step(16)
    assert b.status() == 0
    b.close()


def test_autotune_times_shapes_by_single_steps_also_with_pairs_forced(fake, monkeypatch):
    monkeypatch.setenv("MRLBM_PAIRS", "1")
    s = api.Simulation(large())
    fake.fake_step_us(7, 0.25)
    assert s.autotune(6)[0] == 7
    pairs = fake.fake_done(PAIR)
    s.step(4)
    assert fake.fake_done(PAIR) == pairs + 2                 # and the steps stay paired
    s.close()


@pytest.mark.parametrize("trial_steps", [1, 2, 3, 20])
@pytest.mark.parametrize("loaded", [False, True])
def test_autotune_times_pairs_by_pairs(fake, trial_steps, loaded):
    """Whole pairs, per step: not two single steps against each other, and no single step among them."""
    s = api.Simulation(large())
    if loaded:
        s.load_state(s.get_state(), iter=1)
    fake.fake_reset()
    fake.fake_pair_us(1.9)                                   # single steps take 1 us each
    _, ms = s.autotune(trial_steps)
    assert ms == pytest.approx(0.95e-3, rel=1e-3)
    fake.fake_reset()
    fake.fake_pair_us(2.1)
    _, ms = s.autotune(trial_steps)
    assert ms == pytest.approx(1e-3, rel=1e-3)
    s.close()


@pytest.mark.parametrize("prec", [64, 32])
@pytest.mark.parametrize("loaded", [False, True])
@pytest.mark.parametrize("replayed,chosen", [(0.8, 4), (0.95, 10)])
def test_autotune_times_a_tma_shape_against_replayed_runs(fake, prec, loaded, replayed, chosen):
    """Every shape but the TMA ones is replayed on small lattices; the launched steps of all are timed."""
    s = api.Simulation(small(), precision=prec)
    if loaded:
        s.load_state(s.get_state(), iter=1)
    fake.fake_step_us(4, 0.99)
    fake.fake_step_us(10, 0.9)
    fake.fake_graph_factor(replayed)
    cfg, ms = s.autotune(6)
    assert cfg == chosen and ms == pytest.approx(min(0.9, 0.99 * replayed) * 1e-3, rel=1e-3)
    s.step(300)                                              # the trial's run does not count as asked for
    assert fake.fake_captures() == 1 and s.iter == 301
    s.close()


def test_autotune_keeps_a_tma_shape_where_runs_are_not_replayed(fake):
    cfg = cylinder_case(1003, 403, 60, 250.0, 201.5, 120.0, 0.05)
    s = api.Simulation(cfg, precision=32)
    fake.fake_step_us(10, 0.9)
    fake.fake_pair_us(1e3)
    fake.fake_graph_factor(0.1)
    assert s.autotune(6)[0] == 10
    assert fake.fake_captures() == 0
    s.close()


def test_autotune_without_pairs_when_their_trial_fails(fake):
    s = api.Simulation(large())
    level = s.info.state_bytes // 2
    used = fake.fake_used()
    tuned_pairs(fake)
    fake.fake_fail(b"pair", 1)
    s.autotune(6)
    assert fake.fake_used() < used and s.iter == 1           # single steps, without the third level
    assert used - fake.fake_used() < 2 * level
    s.step(6)
    s.close()


@pytest.mark.parametrize("prec,nodes,calls,captures", [
    (64, "small", [383], 0), (64, "small", [384], 1), (64, "small", [200, 200], 1), (64, "small", [1536], 1),
    (64, "mid", [767], 0), (64, "mid", [768], 1),
    (32, "small", [800], 0), (32, "small", [1535], 0), (32, "small", [1536], 1), (32, "mid", [800], 0),
    # steps of calls too short for a run do not count towards it
    (64, "small", [1] * 5000 + [64], 0), (32, "small", [40] * 50 + [64], 0), (64, "small", [15] * 100 + [300], 0)])
def test_runs_are_captured_once_calls_that_hold_them_pay_for_it(fake, prec, nodes, calls, captures):
    cfg = small() if nodes == "small" else cylinder_case(400, 260, 20, 100.0, 130.5, 100.0, 0.05)
    s = api.Simulation(cfg, precision=prec)
    for n in calls:
        s.step(n)
    assert (fake.fake_captures() > 0) == (captures > 0)
    assert fake.fake_done(STEP) == sum(calls)
    s.close()
