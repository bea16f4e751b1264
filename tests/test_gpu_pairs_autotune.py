"""The autotuner on lattices large enough for it to try pairs: it may switch them on or off without touching the
run, whether they were on by rule before or not."""
import numpy as np
import pytest

from mrlbm_2d_b200.config import cylinder_case

pytestmark = pytest.mark.gpu

# below the size from which pairs are on by rule (700,000 nodes in FP64, 1,500,000 in FP32) and above it
LATTICES = {"off": (1003, 403), "on": (2011, 757)}


@pytest.mark.parametrize("trial_steps", [1, 8])
@pytest.mark.parametrize("prec", [64, 32])
@pytest.mark.parametrize("rule", sorted(LATTICES))
def test_autotuning_a_large_lattice_leaves_the_run(mrlbm, monkeypatch, prec, rule, trial_steps):
    nx, ny = LATTICES[rule]
    cfg = cylinder_case(nx, ny, 60, 250.0, ny // 2 + 0.5, 120.0, 0.05, seed=9, noise=1e-3)
    out, tuning = {}, {}
    for pairs in (None, "0"):
        monkeypatch.setenv("MRLBM_PAIRS", pairs) if pairs else monkeypatch.delenv("MRLBM_PAIRS", raising=False)
        s = mrlbm.Simulation(cfg, precision=prec)
        s.field_stats_window(4, 30)
        s.step(7)
        n = s.launch_count()
        if pairs is None:
            s.autotune(trial_steps)
            tuning[pairs] = s.launch_count() - n
            s.step(20)
        else:
            s.step(20)
            out_plain = [s.get_state(), *s.forces()]
            n = s.launch_count()
            s.autotune(trial_steps)
            tuning[pairs] = s.launch_count() - n
        out[pairs] = out_plain if pairs else [s.get_state(), *s.forces()]
        f = s.field_stats()
        out[pairs] += [f[k] for k in sorted(f)]
        assert s.status() == 0 and s.iter == 28
        s.close()
    for x, y in zip(out[None], out["0"]):
        assert np.array_equal(x, y)
    # the trial of pairs: four steps and an even number of at least two, two launches a pair
    assert tuning[None] - tuning["0"] >= 4 + max(2, trial_steps)
