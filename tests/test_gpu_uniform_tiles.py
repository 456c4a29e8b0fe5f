"""k_blend's packed path (tiles of one camera at weight 256) and the collapsed levels' storage, where they can go
wrong: collapsed values outside the packed range -256 .. 767, uniform tiles on the canvas border and beside
uncovered ones, every output format, odd sizes.  The bytes and the collapsed levels are the oracle's."""
import numpy as np
import pytest

import panostitcher_gb300 as P

pytestmark = pytest.mark.gpu


def _blend(cov, seams, imgs, levels):
    import oracle as O
    import torch
    n, h, w = cov.shape
    b = P.CudaTilingMultibandBlendFast()
    assert b.prepare(list(cov), list(seams), levels, 2)
    ref = O.Blender(cov, seams, levels).blend(list(imgs))
    dev = [torch.from_numpy(np.ascontiguousarray(i)).cuda() for i in imgs]
    for c in (4, 3):
        out = torch.full((h, w, c), 7, dtype=torch.uint8, device="cuda")
        b.blend(dev, out)
        assert np.array_equal(out.cpu().numpy()[..., :3], ref[..., :3])


@pytest.mark.parametrize("w,h", [(256, 96), (449, 131), (640, 352)])
@pytest.mark.parametrize("period", [1, 3, 16])
def test_black_and_white_content(cuda, oracle_lib, w, h, period):
    """Hard black and white: Laplacians of +-255 on every level, so the collapsed values swing far beyond a
    byte and leave the packed range in places."""
    rng = np.random.default_rng([w, h, period])
    cov = np.full((2, h, w), 255, np.uint8)
    cov[0][:, w * 3 // 4:] = 0
    cov[1][:, : w // 4] = 0
    seams = cov.copy()
    seams[0][:, w // 2:] = 0
    seams[1][:, : w // 2] = 0
    y, x = np.mgrid[0:h, 0:w]
    board = (((x // period) + (y // period)) % 2 * 255).astype(np.int16)
    imgs = np.zeros((2, h, w, 4), np.int16)
    for c in range(3):
        imgs[0, ..., c] = board
        imgs[1, ..., c] = np.where(rng.random((h, w)) < 0.5, 255, 0)
    imgs[cov == 0] = 0
    _blend(cov, seams, imgs, 6)


def test_isolated_peaks_leave_the_packed_range(cuda, oracle_lib):
    """Custom masks weight a bright camera's edge against nothing: single white pixels in black and the inverse
    next to coverage holes."""
    rng = np.random.default_rng(5)
    h, w, n = 208, 520, 3
    cov = np.zeros((n, h, w), np.uint8)
    for i in range(n):
        cov[i][:, max(0, i * w // n - 40): (i + 1) * w // n + 40] = 255
    cov[:, 60:110, 200:330] = 0
    seams = np.zeros_like(cov)
    for i in range(n):
        seams[i][:, i * w // n: (i + 1) * w // n] = 255
    seams &= cov
    imgs = np.zeros((n, h, w, 4), np.int16)
    imgs[..., :3] = np.where(rng.random((n, h, w, 1)) < 0.02, 255, 0)
    imgs[1, ..., :3] = 255 - imgs[1, ..., :3]
    imgs[cov == 0] = 0
    _blend(cov, seams, imgs, 8)


@pytest.mark.parametrize("fmt", ["nv12", "yuv420p", "bgr24", "bgr32"])
def test_uniform_tiles_in_every_output_format(cuda, oracle_lib, fmt):
    import oracle as O
    import torch
    from _util import Prepared
    from panostitcher_gb300 import synth as S
    cams = [S.photo_param(1, 200.0, 0.0), S.photo_param(1, 200.0, 180.0)]
    p = Prepared(S.RigConfig("uni", cams, (300, 300), (900, 450), 4, (0.8, 1.2)))
    f = p.frames.frame(0)
    ref = p.oracle_render(f, p.luts)
    dev = [torch.from_numpy(x).cuda() for x in f]
    if fmt.startswith("bgr"):
        c = 4 if fmt == "bgr32" else 3
        store = torch.zeros(4 + 450 * (900 * c + 4), dtype=torch.uint8, device="cuda")
        for shift, pad in ((0, 0), (4, 4)):  # 8-byte aligned rows and rows that are not
            out = store.as_strided((450, 900, c), (900 * c + pad, c, 1), shift)
            p.r.render(dev, out, p.luts, check=True)
            assert np.array_equal(out.cpu().numpy()[..., :3], ref[..., :3])
        return
    planes = [torch.zeros((450, 900), dtype=torch.uint8, device="cuda")]
    planes += ([torch.zeros((225, 900), dtype=torch.uint8, device="cuda")] if fmt == "nv12" else
               [torch.zeros((225, 450), dtype=torch.uint8, device="cuda") for _ in range(2)])
    p.r.render_yuv(dev, planes, p.luts, P.PS_FMT_NV12 if fmt == "nv12" else P.PS_FMT_YUV420P, check=True)
    for a, b in zip(planes, O.bgr32_to_yuv(ref, O.FMT_NV12 if fmt == "nv12" else O.FMT_YUV420P)):
        assert np.array_equal(a.cpu().numpy(), b)
