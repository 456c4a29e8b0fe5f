"""cudaReprojectTo16S where the canvas ends inside a warp's 16x2 pixels, and a canvas of the large build, against the
oracle.  Equal integers."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fmt", ["bgr32", "bgr24"])
@pytest.mark.parametrize("w,h", [(1, 1), (15, 1), (17, 3), (64, 15), (65, 17), (130, 33), (3217, 1601)])
def test_canvas_edges(cuda, oracle_lib, fmt, w, h):
    import oracle as O
    import torch
    from panostitcher_gb300.render import reproject_to_16s
    rng = np.random.default_rng([w, h])
    sw, sh, c = 211, 97, 3 if fmt == "bgr24" else 4
    src = rng.integers(0, 256, (sh, sw, c), dtype=np.uint8)
    xm, ym = ((rng.random((h, w)) * n * 1.25 - n / 8).astype(np.float32) for n in (sw, sh))
    # the last row: every other block invalid throughout, so that lanes of a warp differ in what they skip
    xm[-1, np.arange(w) // 16 % 2 == 1] = -1
    bad = (xm < 0) | (ym < 0) | (xm >= sw) | (ym >= sh)
    xm[bad] = ym[bad] = -1
    lut = rng.integers(0, 256, (3, 256), dtype=np.uint8)
    want = O.reproject_16s(src, xm, ym, lut)
    out = torch.full((h, w, 4), 7, dtype=torch.int16, device="cuda")
    reproject_to_16s(torch.from_numpy(src).cuda(), torch.from_numpy(xm).cuda(), torch.from_numpy(ym).cuda(), out,
                     torch.from_numpy(lut).cuda())
    assert np.array_equal(out.cpu().numpy()[..., :3], want[..., :3])
    assert not out[..., 3].any()
