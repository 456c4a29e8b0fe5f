"""k_pyrdown_pair (two few-tile pyramid levels a launch) where its rule begins and ends (a level of 64x32 under one of
twice its width, one column less), at even and odd heights, with cameras that wrap around the canvas, ragged coverage
and more cameras than the tail kernel takes; and rigs of different depths in one batch.  Equal bytes, no tolerance."""
import numpy as np
import pytest

import panostitcher_gb300 as P

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2, 17])
@pytest.mark.parametrize("w,h", [(128, 64), (126, 64), (128, 63), (130, 95), (256, 65), (320, 130), (262, 257)])
def test_blend_matches_the_oracle(cuda, oracle_lib, w, h, n):
    import oracle as O
    import torch
    rng = np.random.default_rng([w, h, n])
    cov = np.zeros((n, h, w), np.uint8)
    for i in range(n):  # the last camera wraps
        cov[i][:, ((i + 1) * w // n - w // 3 + np.arange(w // 2)) % w] = 255
        cov[i][rng.random((h, w)) < 0.001] = 0
    cov[0, :h // 2] = 255
    best = np.where(cov > 0, rng.random((n, 1, 1)) + 0.3 * rng.random((n, h, w)), -1).argmax(0)
    seams = np.stack([((best == i) & (cov.max(0) > 0)).astype(np.uint8) * 255 for i in range(n)])
    imgs = rng.integers(0, 256, (n, h, w, 4)).astype(np.int16)
    imgs[..., 3] = 0
    imgs[cov == 0] = 0
    b = P.CudaTilingMultibandBlendFast()
    assert b.prepare(list(cov), list(seams), 5, 1), b.last_error
    ref = O.Blender(cov, seams, 5, 1).blend(list(imgs))
    out = torch.zeros((h, w, 4), dtype=torch.uint8, device="cuda")
    b.blend([torch.from_numpy(i).cuda() for i in imgs], out)
    assert np.array_equal(out.cpu().numpy()[..., :3], ref[..., :3])


def test_batch_of_different_depths(cuda):
    import torch
    from _util import Prepared
    from panostitcher_gb300 import synth as S
    cams = [S.photo_param(0, 110.0, 360.0 * k / 4, 0.0) for k in range(4)]
    ps = [Prepared(S.RigConfig("pair", cams, (40, 30), (w, w // 2), lv, (0.8, 1.2)))
          for w, lv in ((256, 8), (132, 3), (520, 4), (1024, 9))]
    frames = [[torch.from_numpy(f).cuda() for f in p.frames.frame(0)] for p in ps]
    ref = [p.product_render(p.frames.frame(0), p.luts) for p in ps]
    dsts = [torch.zeros((p.cfg.dst_size[1], p.cfg.dst_size[0], 4), dtype=torch.uint8, device="cuda") for p in ps]
    P.render_batch([p.r for p in ps], frames, dsts, [p.luts for p in ps])
    torch.cuda.synchronize()
    for d, r in zip(dsts, ref):
        assert np.array_equal(d.cpu().numpy()[..., :3], r[..., :3])
