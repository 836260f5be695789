"""A scene of a batch that has gone non-finite leaves the scenes stored beside it alone: they equal their own runs as the
same steps of a healthy batch do (sums over the particles of a node in another order, 5e-6 of each field's largest
magnitude a step, C's taken as |v| / dx at least)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _scenes(gpe_mod, counts):
    from gpe import scenes

    g = np.random.default_rng(sum(counts))
    p = scenes.mixed_params(1024, 64)
    table, parts = [], []
    for q, n in enumerate(counts):
        nx = 24 + 8 * q
        table.append((nx, nx, (2 * p.dx, 2 * p.dx), ((nx - 3) * p.dx, (nx - 3) * p.dx)))
        # a few particles a node, in the order of their cells
        x = g.uniform(0.4, 0.4 + 0.5 * np.sqrt(n) / nx, (n, 2)) * nx * p.dx
        x = x[np.lexsort(((x[:, 0] / p.dx).astype(int), (x[:, 1] / p.dx).astype(int)))]
        parts.append((x.astype(np.float32), g.normal(0, 0.3, (n, 2)).astype(np.float32),
                      g.normal(0, 1, (n, 4)).astype(np.float32), (g.integers(0, 5, n)).astype(np.int32)))
    return p, table, parts


@pytest.mark.parametrize("counts", [(63, 40, 90), (64, 41, 31), (33, 1, 2), (128, 64, 129)])
@pytest.mark.parametrize("what", ["C nan", "v inf", "v nan"])
@pytest.mark.parametrize("sort_interval", [0, 1])
@pytest.mark.parametrize("calls", [(4,), (1, 1, 1, 1)])
def test_scenes_beside_a_non_finite_one_equal_their_own_runs(gpe_mod, cuda_ok, counts, what, sort_interval, calls):
    p, table, parts = _scenes(gpe_mod, counts)
    p.sort_interval = sort_interval
    x, v, Cm, mat = (np.concatenate([q[k] for q in parts]) for k in range(4))
    sid = np.repeat(np.arange(3), counts).astype(np.int32)
    (Cm if what[0] == "C" else v)[sid == 1] = np.nan if what.endswith("nan") else np.inf
    e = gpe_mod.Mpm(p, capacity=len(x), scenes=[gpe_mod.make_mpm_scene(*t) for t in table])
    e.set_state(x, v, Cm, material=mat, scene_id=sid)
    for c in calls:
        e.step(c)
    got = e.get_state()
    assert e.status() & gpe_mod.STATUS_NONFINITE
    for q in (0, 2):
        solo = gpe_mod.Mpm(p, capacity=counts[q], scenes=[gpe_mod.make_mpm_scene(*table[q])])
        solo.set_state(*parts[q][:3], material=parts[q][3])
        for c in calls:
            solo.step(c)
        assert solo.status() == 0
        want = solo.get_state()
        for f, (a, b) in enumerate(zip(got, want)):
            scale = max(np.abs(b).max(), np.abs(want[1]).max() / p.dx if f == 2 else 0.0)
            assert np.abs(a[sid == q] - b).max() <= 2e-5 * scale, f"scene {q}, field {f}"
