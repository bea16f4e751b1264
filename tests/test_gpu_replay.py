"""Runs of steps replayed from captured graphs (from 384 steps of a handle on 16, from 1536 on 64 at a time) give the bits of steps launched
one call at a time: populations, every force record and field statistics, whatever begins or ends inside a run."""
import numpy as np
import pytest

from cases import CASES, small_reference
from mrlbm_2d_b200.config import cylinder_case

pytestmark = pytest.mark.gpu


def _out(s, fields=False):
    out = [s.get_state(), *s.forces()]
    if fields:
        f = s.field_stats()
        out += [f[k] for k in sorted(f)]
    return out


def _advance(s, n, whole):
    for m in ([n] if whole else [1] * n):
        s.step(m)


def _both(mrlbm, cfg, prec, script):
    outs = []
    for whole in (True, False):
        s = mrlbm.Simulation(cfg, precision=prec)
        outs.append(script(s, lambda n: _advance(s, n, whole)))
        assert s.status() == 0
        s.close()
    assert len(outs[0]) == len(outs[1])
    for x, y in zip(*outs):
        assert np.array_equal(x, y)


@pytest.mark.parametrize("pairs", ["0", "1"])
@pytest.mark.parametrize("prec", [64, 32])
@pytest.mark.parametrize("name", sorted(CASES))
def test_replayed_runs_equal_launched_steps(mrlbm, monkeypatch, prec, pairs, name):
    monkeypatch.setenv("MRLBM_PAIRS", pairs)
    cfg = CASES[name]()
    if cfg.post_process:
        cfg = cfg.replace(statsbegin=50, statsend=2615)        # records begin and end inside runs

    def script(s, go):
        go(2600)                                               # 64, then 16 a run, then single steps
        out = _out(s)
        go(47)                                                 # an odd count: the other time level
        go(64)
        return out + _out(s)

    _both(mrlbm, cfg, prec, script)


@pytest.mark.parametrize("pairs", ["0", "1"])
@pytest.mark.parametrize("prec", [64, 32])
def test_replayed_runs_with_changing_inputs(mrlbm, monkeypatch, prec, pairs):
    monkeypatch.setenv("MRLBM_PAIRS", pairs)
    cfg = CASES["freeslip_label15"]()
    rng = np.random.default_rng(9)
    body = 1e-6 * rng.standard_normal((2, cfg.nx, cfg.ny))
    profile = cfg.uo * (1.0 + 0.1 * rng.standard_normal(cfg.ny))

    def script(s, go):
        go(700)
        out = _out(s)
        s.field_stats_window(740, 840)                         # opens and closes inside runs
        go(160)
        out += _out(s, fields=True)
        s.set_body_force(body)
        s.field_stats_window(861, 10000)
        go(130)
        s.set_inlet_profile(profile)
        go(130)
        out += _out(s, fields=True)
        s.set_body_force(None)
        s.set_inlet_profile(None)
        s.load_state(out[0], iter=30)
        go(70)
        s.surface_enable(True)                                 # launched steps
        go(50)
        s.surface_enable(False)
        go(70)
        s.step(70, macro=True)
        m = s.macro()
        return out + _out(s) + [m[k] for k in sorted(m)]

    _both(mrlbm, cfg, prec, script)


@pytest.mark.parametrize("prec,tile", [(64, 0), (64, 16), (64, 22), (32, 3), (32, 17), (32, 23), (64, 10)])
def test_replayed_runs_of_every_kind_of_tile(mrlbm, prec, tile):
    cfg = small_reference(iplot=40)                            # plot steps inside and outside of runs

    def script(s, go):
        s.tile_config = tile
        go(700)
        return _out(s)

    _both(mrlbm, cfg, prec, script)


def test_replayed_runs_stop_at_a_full_record_ring(mrlbm):
    _both(mrlbm, small_reference(iplot=0), 64, lambda s, go: (go(8300), _out(s))[1])


def test_steps_inside_a_callers_capture_are_launched(mrlbm):
    import torch

    cfg = cylinder_case(120, 48, 12, 30.0, 24.5, 100.0, 0.05, seed=4, noise=1e-2)
    outs = []
    for captured in (True, False):
        st = torch.cuda.Stream()
        s = mrlbm.Simulation(cfg, precision=64)
        s.set_stream(st.cuda_stream)
        s.step(2560)
        s.forces()
        if captured:
            g = torch.cuda.CUDAGraph()
            with torch.cuda.graph(g, stream=st, capture_error_mode="thread_local"):
                s.step(64)
            g.replay()
            torch.cuda.synchronize()
        else:
            s.step(64)
        outs.append(_out(s))
        s.close()
    for x, y in zip(*outs):
        assert np.array_equal(x, y)
