"""Replayed runs of a handle that has been asked for enough steps for every run length it uses (1536 for runs of 64,
384 in FP64 for runs of 16), from then on with changing inputs and shapes: the bits of steps launched one call
at a time."""
import numpy as np
import pytest

from cases import CASES, small_reference

pytestmark = pytest.mark.gpu


def _both(mrlbm, cfg, prec, script):
    outs = []
    for whole in (True, False):
        s = mrlbm.Simulation(cfg, precision=prec)
        outs.append(script(s, lambda n, s=s, whole=whole: [s.step(m) for m in ([n] if whole else [1] * n)]))
        assert s.status() == 0
        s.close()
    for x, y in zip(*outs):
        assert np.array_equal(x, y)


@pytest.mark.parametrize("pairs", ["0", "1"])
@pytest.mark.parametrize("prec", [64, 32])
def test_runs_with_changing_inputs(mrlbm, monkeypatch, prec, pairs):
    monkeypatch.setenv("MRLBM_PAIRS", pairs)
    cfg = CASES["freeslip_label15"]()
    rng = np.random.default_rng(9)
    body = 1e-6 * rng.standard_normal((2, cfg.nx, cfg.ny))
    profile = cfg.uo * (1.0 + 0.1 * rng.standard_normal(cfg.ny))

    def script(s, go):
        go(1600)
        out = [s.get_state(), *s.forces()]
        s.field_stats_window(1640, 1900)                       # opens and closes inside runs
        go(161)
        s.set_body_force(body)
        go(161)
        s.set_inlet_profile(profile)
        go(200)
        f = s.field_stats()
        out += [f[k] for k in sorted(f)] + [s.get_state()]
        s.set_body_force(None)
        s.set_inlet_profile(None)
        s.load_state(out[0], iter=30)
        go(131)
        s.step(130, macro=True)
        m = s.macro()
        return out + [s.get_state(), *s.forces()] + [m[k] for k in sorted(m)]

    _both(mrlbm, cfg, prec, script)


@pytest.mark.parametrize("prec,tile", [(64, 0), (64, 16), (64, 23), (32, 3), (32, 17), (32, 23)])
def test_runs_of_every_kind_of_tile(mrlbm, prec, tile):
    def script(s, go):
        s.tile_config = tile
        go(1700)
        return [s.get_state(), *s.forces()]

    _both(mrlbm, small_reference(iplot=200), prec, script)
