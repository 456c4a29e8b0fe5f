"""Explicit seams that reach beyond the cameras' coverage: whole 64x16 tiles of one camera's seam that no camera
covers, and tiles that one covers in part.  Uncovered pixels are 0 in every output, and all bytes are the oracle's,
on both sides of the line between k_blend_rows and k_blend."""
import numpy as np
import pytest

import panostitcher_gb300 as P

pytestmark = pytest.mark.gpu


def _uniform_tiles(cov, seams):
    """How many level-0 tiles are one camera's seam throughout, by what is covered of them: nothing, a part."""
    none = part = 0
    n, h, w = cov.shape
    union = cov.max(0) > 0
    for y in range(0, h, 16):
        for x in range(0, w, 64):
            if (seams[:, y:y + 16, x:x + 64] > 0).all((1, 2)).any():
                u = union[y:y + 16, x:x + 64]
                none += not u.any()
                part += bool(u.any() and not u.all())
    return none, part


# 220 tiles (k_blend_rows), 2880 (k_blend), 2990 with ragged edges
@pytest.mark.parametrize("w,h", [(640, 352), (2880, 1024), (2881, 1037)])
@pytest.mark.parametrize("levels", [1, 4])
def test_blender(cuda, oracle_lib, w, h, levels):
    import oracle as O
    import torch
    cov = np.zeros((2, h, w), np.uint8)
    cov[0][h // 8: h * 5 // 8 + 5, w // 10: w // 2 + 30] = 255
    cov[1][h // 8: h * 5 // 8 + 5, w // 2 - 30: w * 9 // 10 + 3] = 255
    seams = np.zeros_like(cov)
    seams[0][:, : w // 2] = 255
    seams[1][:, w // 2:] = 255
    assert min(_uniform_tiles(cov, seams)) > 0
    rng = np.random.default_rng([w, h, levels])
    imgs = rng.integers(0, 256, (2, h, w, 4)).astype(np.int16)
    imgs[..., 3] = 0
    imgs[cov == 0] = 0
    ref = O.Blender(cov, seams, levels).blend(list(imgs))[..., :3]
    assert not ref[cov.max(0) == 0].any()
    b = P.CudaTilingMultibandBlendFast()
    assert b.prepare(list(cov), list(seams), levels, 2), b.last_error
    dev = [torch.from_numpy(i).cuda() for i in imgs]
    for c in (4, 3):
        out = torch.full((h, w, c), 7, dtype=torch.uint8, device="cuda")
        b.blend(dev, out)
        assert np.array_equal(out.cpu().numpy()[..., :3], ref)


@pytest.mark.parametrize("dst", [640, 2880])
def test_render(cuda, oracle_lib, dst):
    import oracle as O
    import torch
    from _util import Prepared
    from panostitcher_gb300 import synth as S
    h, w = dst // 2, dst
    cams = [S.photo_param(1, 130.0, 0.0), S.photo_param(1, 130.0, 180.0)]
    col = np.arange(w)
    front = np.broadcast_to((col >= w // 4) & (col < w * 3 // 4), (h, w))
    seams = [np.ascontiguousarray(np.where(m, 255, 0), dtype=np.uint8) for m in (front, ~front)]
    p = Prepared(S.RigConfig("gap", cams, (300, 300), (w, h), 4, (0.8, 1.2)), seams=seams)
    assert min(_uniform_tiles(p.cov, np.stack(seams))) > 0
    f = p.frames.frame(0)
    ref = p.oracle_render(f, p.luts, nthreads=8)
    dev = [torch.from_numpy(x).cuda() for x in f]
    out = torch.full((h, w, 4), 7, dtype=torch.uint8, device="cuda")
    p.r.render(dev, out, p.luts, check=True)
    assert np.array_equal(out.cpu().numpy()[..., :3], ref[..., :3])
    planes = [torch.zeros((h, w), dtype=torch.uint8, device="cuda"), torch.zeros((h // 2, w), dtype=torch.uint8, device="cuda")]
    p.r.render_yuv(dev, planes, p.luts, P.PS_FMT_NV12, check=True)
    for a, b in zip(planes, O.bgr32_to_yuv(ref, O.FMT_NV12)):
        assert np.array_equal(a.cpu().numpy(), b)
