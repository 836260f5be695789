"""Cell starts at the edges of the scan: cell counts with every remainder of four, around the tiles of 2,048 cells, with
arrays that are and are not 16-byte aligned, and around the tile counts at which the tiles' sums get their own launch;
and scene ids refused wherever in a thread's entries the fault is. Whole numbers: equal."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _points(nx, ny, h, n, seed):
    """n points in cells picked at random, the last cell among them"""
    g = np.random.default_rng(seed)
    ix, iy = g.integers(0, nx, n), g.integers(0, ny, n)
    ix[0], iy[0] = nx - 1, ny - 1
    return (np.stack([ix + 0.5, iy + 0.5], 1) * h).astype(np.float32)


def _params():
    from gpe import scenes

    p = scenes.dam_params(iters=1)
    p.h, p.cell, p.wall_margin, p.dt = 1.0, 0.0, 0.25, 1e-3
    return p


@pytest.mark.parametrize("cells", [(1, 1), (2, 1), (3, 1), (7, 3), (2047, 1), (2048, 1), (2049, 1), (89, 46), (45, 91)])
@pytest.mark.parametrize("offset", [0, 1])
def test_caller_arrays(gpe_mod, cuda_ok, cells, offset):
    import torch

    from test_zz_no_alloc import _fn

    nx, ny = cells
    p, n, m = _params(), 3000, nx * ny
    pos = torch.from_numpy(_points(nx, ny, 1.0, n, m)).cuda()
    vel = torch.zeros_like(pos)
    o_pos, o_pred = torch.empty_like(pos), torch.empty_like(pos)
    key, perm = (torch.empty(n, dtype=torch.int32, device="cuda") for _ in range(2))
    start = torch.full((m + 1 + offset + 8,), -7, dtype=torch.int32, device="cuda")
    dom = gpe_mod.make_domains([(0.0, 0.0, float(nx), float(ny))])
    torch.cuda.synchronize()
    for _ in range(2):  # the second call finds the scratch as the first one's scan left it
        rc = _fn(gpe_mod)(C.byref(p), dom, pos.data_ptr(), vel.data_ptr(), n, o_pos.data_ptr(), o_pred.data_ptr(),
                          key.data_ptr(), perm.data_ptr(), start.data_ptr() + 4 * offset, m, None)
        gpe_mod.check(rc, "gpe_pbf_predict_sort_noalloc")
        torch.cuda.synchronize()
        got = start.cpu().numpy()
        k = key.cpu().numpy()
        xy = o_pos.cpu().numpy().astype(np.int64)
        np.testing.assert_array_equal(k, xy[:, 1] * nx + xy[:, 0])
        want = np.concatenate([[0], np.cumsum(np.bincount(k, minlength=m))])
        np.testing.assert_array_equal(got[offset:offset + m + 1], want)
        assert (got[:offset] == -7).all() and (got[offset + m + 1:] == -7).all()  # nothing beside the array


@pytest.mark.parametrize("cells", [(2049, 2048), (2897, 2895), (2897, 2897)])
def test_many_tiles(gpe_mod, cuda_ok, cells):
    nx, ny = cells
    pos = _points(nx, ny, 1.0, 5000, nx)
    e = gpe_mod.Pbf(_params(), [(0.0, 0.0, float(nx), float(ny))], capacity=len(pos))
    e.set_state(pos, np.zeros_like(pos))
    e.stage(gpe_mod.PBF_STAGE_PREDICT_SORT)
    k = e.field(gpe_mod.PBF_FIELD_KEY)
    assert k.max() == nx * ny - 1
    want = np.concatenate([[0], np.cumsum(np.bincount(k, minlength=nx * ny))])
    np.testing.assert_array_equal(e.field(gpe_mod.PBF_FIELD_CELL_START), want)


@pytest.mark.parametrize("n", [1, 2, 1023, 1024, 1025, 3000])
def test_bad_scene_ids_are_refused(gpe_mod, cuda_ok, n):
    import torch

    boxes = [(0.0, 0.0, 4.0, 4.0), (8.0, 0.0, 4.0, 4.0)]
    pos = torch.full((n, 2), 1.5, device="cuda")
    ok = torch.zeros(n, dtype=torch.int32, device="cuda")
    e = gpe_mod.Pbf(_params(), boxes, capacity=n)
    e.set_state(pos, pos * 0, domain=ok)
    for at in sorted({0, 255, 256, 511, 512, 1023, 1024, n - 2, n - 1}):
        if not 0 <= at < n:
            continue
        for bad in (-1, 2, 1):
            if bad == 1 and at == n - 1:
                continue  # the last particle alone in scene 1 is in order
            dom = ok.clone()
            dom[at] = bad
            with pytest.raises(gpe_mod.GpeError):
                e.set_state(pos, pos * 0, domain=dom)
    e.set_state(pos, pos * 0, domain=ok)
    e.step(1)
    assert e.status() == 0
