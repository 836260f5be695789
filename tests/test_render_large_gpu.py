"""A frame of more than 2^32 pixels: every centre count starts from zero, whatever the scratch held before, with the
scratch on a 16-byte boundary and off it."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("offset", [1, 4])
def test_counts_of_a_frame_beyond_2_to_32_pixels_are_cleared(gpe_mod, cuda_ok, offset):
    torch = pytest.importorskip("torch")
    torch.cuda.empty_cache()
    w, h = 65536, 65537
    if torch.cuda.mem_get_info()[0] < 48 << 30:
        pytest.skip("needs 35 GB of device memory")
    cover = torch.full((w * h + offset,), 3, dtype=torch.int32, device="cuda")
    img = torch.empty(w * h, dtype=torch.int32, device="cuda")
    pos, n = torch.zeros(8, 2, device="cuda"), torch.zeros(1, dtype=torch.int32, device="cuda")
    view = gpe_mod.View(pos.data_ptr(), pos.data_ptr(), n.data_ptr(), 1, 1, 1000.0, 8)
    gpe_mod.render_frame(gpe_mod.Raster(img.data_ptr(), 4 * w, w, h, 1.0, 1000.0, cover[offset:].data_ptr()), view)
    torch.cuda.synchronize()
    counts = cover[offset:]
    assert all(int(counts[i:i + (1 << 28)].max()) == 0 for i in range(0, w * h, 1 << 28))
    # rows without a grid line differ from pixel to pixel only at the lines, which repeat with chunk_dim
    for y in (1, h - 1):
        row = img[y * w:(y + 1) * w]
        assert len(torch.unique(row)) == 2 and int((row != row[1]).sum()) == -(-w // 1000)
    del cover, img, counts
    torch.cuda.empty_cache()
