"""Parameters changed between the stages of a step: the passes after the change use the new radius with lists as without
them, bit for bit (lists made with the old radius lack candidates of a larger one)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("h", [0.018, 0.0225, 0.03])
def test_radius_changed_between_stages(gpe_mod, cuda_ok, h):
    from gpe import scenes

    pos, _, boxes = scenes.dam_break(n_side=64)
    vel = np.random.default_rng(3).normal(0, 0.2, pos.shape).astype(np.float32)
    got = []
    for skin in (0.075, 0.0):
        p = scenes.dam_params(iters=2)
        p.dt, p.cell = 1.0 / 480.0, p.h
        e = gpe_mod.Pbf(p, boxes, capacity=len(pos))
        e.set_tuning(cell=p.h, skin=skin)
        e.set_state(pos, vel)
        e.stage(gpe_mod.PBF_STAGE_PREDICT_SORT)
        e.stage(gpe_mod.PBF_STAGE_LAMBDA)
        p.h = h
        e.set_params(p)
        for stage in (gpe_mod.PBF_STAGE_DELTA_P, gpe_mod.PBF_STAGE_LAMBDA, gpe_mod.PBF_STAGE_DELTA_P):
            e.stage(stage)
        got.append((e.field(gpe_mod.PBF_FIELD_LAMBDA), e.field(gpe_mod.PBF_FIELD_DISP)))
    for a, b in zip(*got):
        np.testing.assert_array_equal(a, b)
