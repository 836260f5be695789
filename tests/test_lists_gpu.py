"""Candidate lists at the edges of what they hold: scenes wide enough for 32-bit slots, rows so full that the next
row's slots lie further away than a 16-bit slot reaches, and particle counts around the groups of four that the
scans take. The state after the steps equals the full scans' bit for bit (a list leaves out only exact zeros)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _scene(kind):
    from gpe import scenes

    p = scenes.dam_params(iters=3)
    p.dt = 1.0 / 480.0
    if kind == "wide":  # 4,200 cells across: 32-bit slots
        nx, ny, spacing, box = 8300, 6, 0.01, (0.0, 0.0, 84.0, 0.4)
    elif kind == "reach":  # 3,900 cells across at about 9 particles a cell: 35,000 slots a row of cells
        nx, ny, spacing, box = 11600, 7, 0.0067, (0.0, 0.0, 78.0, 0.4)
    else:  # a handful of particles
        nx, ny, spacing, box = int(kind), 1, 0.01, (0.0, 0.0, 0.4, 0.4)
    ix, iy = np.meshgrid(np.arange(nx), np.arange(ny))
    pos = np.stack([(ix.ravel() + 0.5) * spacing, (iy.ravel() + 0.5) * spacing], 1)
    g = np.random.default_rng(8)
    pos = (pos + g.uniform(-0.001, 0.001, pos.shape)).astype(np.float32)
    return p, pos, g.normal(0, 0.3, pos.shape).astype(np.float32), [box]


@pytest.mark.parametrize("kind", ["wide", "reach", "1", "2", "5", "33"])
@pytest.mark.parametrize("persistent", [0, 2])
def test_lists_equal_full_scans(gpe_mod, cuda_ok, kind, persistent):
    p, pos, vel, boxes = _scene(kind)
    outs = []
    for skin in (0.0, 0.075):
        e = gpe_mod.Pbf(p, boxes, capacity=len(pos))
        e.set_tuning(skin=skin, persistent=persistent if skin else 0)
        e.set_state(pos, vel)
        e.step(3)
        assert e.status() == 0
        outs.append(e.get_state()[:2])
    for a, b in zip(*outs):
        np.testing.assert_array_equal(a, b)
