"""Two steps per launch pair (MRLBM_PAIRS=1) give the bits of single steps: populations, every force
record, field statistics, on lattices whose strips and chunks of rows end in every remainder, and
the FP64 form meets the oracle."""
import numpy as np
import pytest

from cases import CASES
from mrlbm_2d_b200.config import cylinder_case

pytestmark = pytest.mark.gpu

# (nx - 4) % 30 at 0, 1 and 29, one strip more and fewer than a block's; ny - 4 below and above one chunk
SIZES = [(64, 40), (124, 45), (125, 67), (153, 50), (244, 61), (245, 128), (304, 97)]


def _run(mrlbm, monkeypatch, pairs, cfg, prec, steps, fields=None, body=None):
    monkeypatch.setenv("MRLBM_PAIRS", "1" if pairs else "0")
    s = mrlbm.Simulation(cfg, precision=prec)
    if fields:
        s.field_stats_window(*fields)
    if body is not None:
        s.set_body_force(body)
    n0 = s.launch_count()
    for n in steps:
        s.step(n)
    out = [s.get_state(), *s.forces()]
    if fields:
        f = s.field_stats()
        out += [f[k] for k in sorted(f)]
    s.step(4, macro=True)
    m = s.macro()
    out += [m[k] for k in sorted(m)] + [s.get_state()]
    assert s.status() == 0
    launches = s.launch_count() - n0
    s.close()
    return out, launches


def _same(a, b):
    for x, y in zip(a[0], b[0]):
        assert np.array_equal(x, y)


@pytest.mark.parametrize("prec", [64, 32])
@pytest.mark.parametrize("nx,ny", SIZES)
def test_pairs_equal_single_steps(mrlbm, monkeypatch, prec, nx, ny):
    cfg = cylinder_case(nx, ny, 10, nx // 3, ny // 2 + 0.5, 80.0, 0.05, seed=nx, noise=1e-2)
    _same(_run(mrlbm, monkeypatch, True, cfg, prec, [7, 2, 16]), _run(mrlbm, monkeypatch, False, cfg, prec, [7, 2, 16]))


@pytest.mark.parametrize("prec", [64, 32])
@pytest.mark.parametrize("name", sorted(CASES))
def test_pairs_equal_single_steps_on_every_case(mrlbm, monkeypatch, prec, name):
    cfg = CASES[name]()                             # every closure, wall and periodic option; plot steps
    _same(_run(mrlbm, monkeypatch, True, cfg, prec, [9, 14]), _run(mrlbm, monkeypatch, False, cfg, prec, [9, 14]))


@pytest.mark.parametrize("prec", [64, 32])
def test_pairs_with_field_statistics_and_body_force(mrlbm, monkeypatch, prec):
    cfg = CASES["freeslip_label15"]()
    body = 1e-6 * np.random.default_rng(5).standard_normal((2, cfg.nx, cfg.ny))
    for kw in (dict(fields=(5, 18)), dict(fields=(4, 17), body=body), dict(body=body)):
        _same(_run(mrlbm, monkeypatch, True, cfg, prec, [20], **kw), _run(mrlbm, monkeypatch, False, cfg, prec, [20], **kw))


def test_pairs_meet_the_oracle(mrlbm, oracle_mod, monkeypatch):
    cfg = cylinder_case(185, 76, 14, 60, 38.5, 90.0, 0.05, seed=3, noise=1e-2)
    out, launches = _run(mrlbm, monkeypatch, True, cfg, 64, [30])
    o = oracle_mod.Oracle(cfg)
    o.step(30)
    assert np.array_equal(out[0], o.field("f"))
    for x, y in zip(out[1:5], o.forces()):
        assert np.array_equal(x, y)
    o.close()
    # 15 pairs and the record sums the history read asks for; then a pair and two single steps
    assert launches >= 2 * 15 + 1


@pytest.mark.parametrize("prec", [64, 32])
def test_pairs_after_a_loaded_state_and_autotune(mrlbm, monkeypatch, prec):
    """A loaded state replaces the ghost ring every level carries, and the autotuner may switch pairs on or off
    without touching the run."""
    cfg = CASES["reference_walls"]()
    rng = np.random.default_rng(7)
    res = []
    for pairs in ("1", "0"):
        monkeypatch.setenv("MRLBM_PAIRS", pairs)
        s = mrlbm.Simulation(cfg, precision=prec)
        f0 = s.get_state()
        s.step(5)
        g = f0 * (1.0 + 1e-3 * np.random.default_rng(7).standard_normal(f0.shape))
        s.load_state(g, iter=3)
        s.step(12)
        res.append(s.get_state())
        s.close()
    assert np.array_equal(res[0], res[1])
    monkeypatch.delenv("MRLBM_PAIRS")
    big = cylinder_case(400, 120, 20, 100, 60.5, 100.0, 0.05, seed=int(rng.integers(1000)))
    s, t = mrlbm.Simulation(big, precision=prec), mrlbm.Simulation(big, precision=prec)
    s.step(3)
    s.autotune(trial_steps=4)
    s.step(8)
    t.step(11)
    assert np.array_equal(s.get_state(), t.get_state()) and np.array_equal(s.forces()[1], t.forces()[1])
    s.close()
    t.close()


@pytest.mark.parametrize("prec", [64, 32])
def test_pairs_over_a_long_run_of_full_waves(mrlbm, monkeypatch, prec):
    """Every block resident at once and several rounds of them: a copy that overtakes the reads of its
    ring slot, or a block that starts before the level it reads is complete, shows here and not on
    small lattices."""
    from mrlbm_2d_b200.config import case_mid
    res = []
    for pairs in ("1", "0"):
        monkeypatch.setenv("MRLBM_PAIRS", pairs)
        s = mrlbm.Simulation(case_mid(), precision=prec)
        for _ in range(4):
            s.step(150)
        assert s.status() == 0
        res.append((s.get_state(), s.forces()))
        s.close()
    assert np.array_equal(res[0][0], res[1][0])
    for x, y in zip(res[0][1], res[1][1]):
        assert np.array_equal(x, y)


@pytest.mark.parametrize("prec", [64, 32])
def test_batch_streams_in_pairs(mrlbm, monkeypatch, prec):
    """Per-case streams with the steps in pairs, odd and even call lengths, against each case alone."""
    cfgs = [CASES[n]() for n in ("freeslip_label15", "reference_default_bcs", "reference_walls")]
    cfgs.append(cylinder_case(256, 64, 12.8, 51.2, 32.5, 150.0, 0.05))
    monkeypatch.setenv("MRLBM_PAIRS", "1")
    b = mrlbm.Batch(cfgs, precision=prec)
    b.set_schedule(9, mrlbm.BATCH_STREAMS, 6)
    for n in (6, 12, 9, 5):                         # whole graphs, both start levels, remainders
        b.step(n)
    b.step(7, macro=True)
    assert b.status() == 0
    monkeypatch.setenv("MRLBM_PAIRS", "0")
    for cfg, c in zip(cfgs, b.cases):
        s = mrlbm.Simulation(cfg, precision=prec)
        s.step(39, macro=True)
        assert np.array_equal(c.get_state(), s.get_state())
        for x, y in zip(c.forces(), s.forces()):
            assert np.array_equal(x, y)
        assert np.array_equal(c.macro()["ux"], s.macro()["ux"])
        s.close()
    b.close()


@pytest.mark.parametrize("prec", [64, 32])
def test_pairs_refuse_the_shapes_single_steps_refuse(mrlbm, monkeypatch, prec):
    cfg = cylinder_case(124, 45, 10, 41, 22.5, 80.0, 0.05, seed=2, noise=1e-2)
    seen = []
    for pairs in ("0", "1"):
        monkeypatch.setenv("MRLBM_PAIRS", pairs)
        s = mrlbm.Simulation(cfg, precision=prec)
        refused = []
        for tile in range(mrlbm.N_TILE_CONFIGS):
            s.tile_config = tile
            for n in (2, 5):
                try:
                    s.step(n)
                except mrlbm.MrlbmError:
                    refused.append((tile, n))
        seen.append((refused, s.iter, s.get_state()))
        s.close()
    assert seen[0][:2] == seen[1][:2] and np.array_equal(seen[0][2], seen[1][2])
