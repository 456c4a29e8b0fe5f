"""The blender's input images at the widths and heights where a warp's columns and a thread's rows end, at any row
alignment: one fully covered image blends to itself, whatever lies in the padding of its rows, and a value out of
range or outside the coverage is refused wherever it is."""
import numpy as np
import pytest

import panostitcher_gb300 as P

pytestmark = pytest.mark.gpu


def _prepared(cov):
    b = P.CudaTilingMultibandBlendFast()
    assert b.prepare([cov], [cov], 3)
    return b


@pytest.mark.parametrize("dtype", ["int16", "uint8"])
@pytest.mark.parametrize("w,h", [(1, 1), (31, 2), (33, 3), (127, 5), (129, 4), (513, 7), (640, 2)])
@pytest.mark.parametrize("pad", [0, 1, 3])
def test_images_to_level0(cuda, dtype, w, h, pad):
    import torch
    rng = np.random.default_rng([w, h, pad])
    # the padding and the fourth channel hold values that would be refused in the image
    buf = np.full((h, w + pad, 4), 255 if dtype == "uint8" else -7, dtype)
    buf[:, :w, :3] = rng.integers(0, 256, (h, w, 3))
    b = _prepared(np.full((h, w), 255, np.uint8))
    out = torch.zeros((h, w, 4), dtype=torch.uint8, device="cuda")
    dev = torch.from_numpy(buf).cuda()
    b.blend([dev[:, :w]], out)
    assert np.array_equal(out.cpu().numpy()[..., :3], buf[:, :w, :3].astype(np.uint8))
    if dtype == "uint8":
        return
    for y, x, c in [(0, 0, 0), (h - 1, w - 1, 2), (h // 2, w // 2, 1)]:
        for v in (-1, 256, -32768, 32767):
            bad = dev.clone()
            bad[y, x, c] = v
            with pytest.raises(P.PsError) as e:
                b.blend([bad[:, :w]], out)
            assert e.value.code == P._lib.PS_EINVAL and "0..255" in str(e.value)


@pytest.mark.parametrize("dtype", ["int16", "uint8"])
@pytest.mark.parametrize("w,h", [(33, 3), (129, 4)])
def test_pixels_outside_the_coverage_are_refused(cuda, dtype, w, h):
    import torch
    for y, x in [(0, 0), (h - 1, w - 1), (1, 32)]:
        cov = np.full((h, w), 255, np.uint8)
        cov[y, x] = 0
        b = _prepared(cov)
        out = torch.zeros((h, w, 4), dtype=torch.uint8, device="cuda")
        img = np.full((h, w, 4), 9, dtype)
        img[y, x, :3] = 0  # the fourth channel does not count
        b.blend([torch.from_numpy(img).cuda()], out)
        for c in range(3):
            img[y, x] = 0
            img[y, x, c] = 1
            with pytest.raises(P.PsError) as e:
                b.blend([torch.from_numpy(img).cuda()], out)
            assert e.value.code == P._lib.PS_EINVAL and "coverage" in str(e.value)
