"""Field statistics of steps taken in pairs on lattices whose blocks fill the GPU: the first launch of a pair adds
to the sums of the edges and the cylinder's surroundings while the second one's tiles read their neighbours', so a
sum read from an older copy of its sector would lose a step.  Small lattices never have both at work at once."""
import numpy as np
import pytest

from mrlbm_2d_b200.config import case_mid, cylinder_case

pytestmark = pytest.mark.gpu

LATTICES = {"mid": case_mid, "ragged": lambda: cylinder_case(1531, 613, 96, 300.0, 306.5, 150.0, 0.05, seed=6, noise=1e-3)}


@pytest.mark.parametrize("force", [False, True])
@pytest.mark.parametrize("prec", [64, 32])
@pytest.mark.parametrize("name", sorted(LATTICES))
def test_field_sums_of_pairs_at_full_residency(mrlbm, monkeypatch, prec, name, force):
    cfg = LATTICES[name]()
    res = []
    for pairs in ("1", "0"):
        monkeypatch.setenv("MRLBM_PAIRS", pairs)
        s = mrlbm.Simulation(cfg, precision=prec)
        if force:
            s.set_body_force(1e-7 * np.random.default_rng(8).standard_normal((2, cfg.nx, cfg.ny)))
        s.field_stats_window(2, 1 << 30)
        n0 = s.launch_count()
        for _ in range(3):
            s.step(100)
        launches = s.launch_count() - n0
        assert s.status() == 0
        f = s.field_stats()
        res.append((launches, [f[k] for k in sorted(f)] + [s.get_state(), *s.forces()]))
        s.close()
    assert res[0][0] == 300                                 # 150 pairs of two launches
    for x, y in zip(res[0][1], res[1][1]):
        assert np.array_equal(x, y)
