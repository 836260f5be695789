"""The rasteriser at sizes around its threads' 4 x 4 pixels, its blocks and their rows, with image rows that are and are
not 16-byte aligned (two forms of the shading kernel): the oracle's image byte for byte."""
import numpy as np
import pytest

from test_render_gpu import _raster, _view_from

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("width", [1, 3, 4, 127, 128, 132, 641])
@pytest.mark.parametrize("height", [1, 2, 31, 37])
@pytest.mark.parametrize("pad", [0, 4])
def test_image_sizes(gpe_mod, cuda_ok, oracle, width, height, pad):
    torch = pytest.importorskip("torch")
    g = np.random.default_rng(width * 100 + height)
    scale, dim, cap = 1.7, 9.0, 400
    pos = np.stack([g.uniform(-3, width / scale + 3, (4, cap)), g.uniform(-3, height / scale + 3, (4, cap))], -1)
    pos = pos.astype(np.float32)
    counts = np.array([cap, 0, 7, cap + 5], np.int32)
    view, keep = _view_from(gpe_mod, torch, pos.reshape(-1, 2), counts, 2, 2, dim, cap)
    r, img, cov = _raster(gpe_mod, torch, width, height, scale, dim, pad=pad)
    for _ in range(2):  # the second frame finds the first one's counts in the scratch
        gpe_mod.render_frame(r, view)
    got = img[:, : 4 * width].cpu().numpy().reshape(height, width, 4)
    np.testing.assert_array_equal(got, oracle.render_frame(width, height, scale, dim, pos, counts))
    assert not img[:, 4 * width:].any()  # nothing is written past a row's end
