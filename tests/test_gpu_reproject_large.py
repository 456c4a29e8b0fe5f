"""cudaReprojectTo16S on canvases large enough for its second build: the whole canvas in one call equals its parts in
calls of the other build, which other tests hold against the oracle.  Equal integers."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fmt", ["bgr32", "bgr24", "one column"])
@pytest.mark.parametrize("w,h", [(3200, 1600), (3201, 1999)])
def test_whole_canvas_equals_its_parts(cuda, fmt, w, h):
    import torch
    from panostitcher_gb300.render import reproject_to_16s
    rng = np.random.default_rng([w, h])
    sw, sh = (1, 37) if fmt == "one column" else (611, 407)
    src = torch.from_numpy(rng.integers(0, 256, (sh, sw, 3 if fmt == "bgr24" else 4), dtype=np.uint8)).cuda()
    y, x = np.mgrid[0:h, 0:w].astype(np.float32)
    xm = (x * np.float32(sw / w * 1.1) - np.float32(sw * 0.05) + y * np.float32(0.003)).astype(np.float32)
    ym = (y * np.float32(sh / h * 1.1) - np.float32(sh * 0.05) + x * np.float32(0.001)).astype(np.float32)
    xm[::7, ::5] = np.floor(xm[::7, ::5]) + np.float32(0.5)  # exact ties
    bad = (xm < 0) | (ym < 0) | (xm >= sw) | (ym >= sh)
    xm[bad] = ym[bad] = -1
    xm, ym = torch.from_numpy(xm).cuda(), torch.from_numpy(ym).cuda()
    lut = torch.from_numpy(rng.integers(0, 256, (3, 256), dtype=np.uint8)).cuda()
    whole = torch.full((h, w, 4), 7, dtype=torch.int16, device="cuda")
    parts = torch.full((h, w, 4), 9, dtype=torch.int16, device="cuda")
    reproject_to_16s(src, xm, ym, whole, lut)
    for r in range(0, h, 400):
        reproject_to_16s(src, xm[r:r + 400], ym[r:r + 400], parts[r:r + 400], lut)
    torch.cuda.synchronize()
    assert torch.equal(whole, parts)
    assert bool((whole[..., :3] != 0).any())
