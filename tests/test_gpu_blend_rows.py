"""k_blend and k_blend_rows on either side of the line between them, and k_blend_rows with one and two row pairs a
warp: collapsed values outside the packed range, odd sizes, uncovered tiles, tiles of many cameras, levels above 0
(small_blend_max_items 1 hands them all to these kernels), every output format.  Equal bytes, no tolerance."""
import numpy as np
import pytest

import panostitcher_gb300 as P

pytestmark = pytest.mark.gpu


# tiles of 64x16: 8, 931, 1995, 2665 (k_blend), 2706 with a ragged edge (k_blend)
@pytest.mark.parametrize("w,h", [(253, 31), (1217, 771), (2240, 900), (2624, 1040), (2625, 1041)])
def test_black_and_white_content(cuda, oracle_lib, w, h):
    import oracle as O
    import torch
    rng = np.random.default_rng([w, h])
    n = 3
    cov = np.full((n, h, w), 255, np.uint8)
    cov[0][:, w * 3 // 4:] = 0
    cov[1][:, : w // 4] = 0
    cov[2][: h // 2] = 0
    cov[:, h // 5: h // 3, w // 8: w // 6] = 0
    seams = cov.copy()
    seams[0][:, w // 2:] = 0
    seams[1][:, : w // 2] = 0
    seams[2] = 0
    seams[2][h * 7 // 8:] = cov[2][h * 7 // 8:]
    seams[:2, h * 7 // 8:] = 0
    y, x = np.mgrid[0:h, 0:w]
    imgs = np.zeros((n, h, w, 4), np.int16)
    imgs[0, ..., :3] = (((x // 3) + (y // 3)) % 2 * 255)[..., None]
    imgs[1, ..., :3] = np.where(rng.random((h, w, 1)) < 0.5, 255, 0)
    imgs[2, ..., :3] = rng.integers(0, 256, (h, w, 3))
    imgs[cov == 0] = 0
    b = P.CudaTilingMultibandBlendFast()
    assert b.prepare(list(cov), list(seams), 5, 2), b.last_error
    ref = O.Blender(cov, seams, 5).blend(list(imgs))
    dev = [torch.from_numpy(i).cuda() for i in imgs]
    for c in (4, 3):
        out = torch.full((h, w, c), 7, dtype=torch.uint8, device="cuda")
        b.blend(dev, out)
        assert np.array_equal(out.cpu().numpy()[..., :3], ref[..., :3])


@pytest.mark.parametrize("dst,n", [(260, 11), (900, 2), (2656, 2)])
@pytest.mark.parametrize("fmt", ["nv12", "yuv420p", "bgr24"])
def test_levels_and_output_formats(cuda, oracle_lib, dst, n, fmt):
    import oracle as O
    import torch
    from _util import Prepared
    from panostitcher_gb300 import synth as S
    cams = [S.photo_param(1, 200.0, 360.0 * k / n) for k in range(n)]
    p = Prepared(S.RigConfig("rows", cams, (300, 300), (dst, dst // 2), 4, (0.8, 1.2)))
    p.r.set_launch_shape(tail_max_items=0, small_blend_max_items=1)
    f = p.frames.frame(0)
    ref = p.oracle_render(f, p.luts, nthreads=8)
    dev = [torch.from_numpy(x).cuda() for x in f]
    h, w = dst // 2, dst
    if fmt == "bgr24":
        out = torch.zeros((h, w, 3), dtype=torch.uint8, device="cuda")
        p.r.render(dev, out, p.luts, check=True)
        assert np.array_equal(out.cpu().numpy(), ref[..., :3])
        return
    planes = [torch.zeros((h, w), dtype=torch.uint8, device="cuda")]
    planes += ([torch.zeros((h // 2, w), dtype=torch.uint8, device="cuda")] if fmt == "nv12" else
               [torch.zeros((h // 2, w // 2), dtype=torch.uint8, device="cuda") for _ in range(2)])
    p.r.render_yuv(dev, planes, p.luts, P.PS_FMT_NV12 if fmt == "nv12" else P.PS_FMT_YUV420P, check=True)
    for a, b in zip(planes, O.bgr32_to_yuv(ref, O.FMT_NV12 if fmt == "nv12" else O.FMT_YUV420P)):
        assert np.array_equal(a.cpu().numpy(), b)
