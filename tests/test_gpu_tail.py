"""The few-tile levels (k_tail, k_blend_small) at the sizes where their tiles and footprints go wrong: levels
narrower than a footprint, odd sizes, one-pixel levels, more cameras than a unit stages, whole tiles, several
units per CTA.  Every shape gives the oracle's bytes."""
import numpy as np
import pytest

import panostitcher_gb300 as P

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h,n", [(2, 1, 1), (3, 2, 2), (33, 17, 3), (65, 15, 2), (66, 34, 9), (127, 63, 17),
                                   (200, 100, 4), (513, 40, 8)])
def test_blender_levels_match_the_oracle(cuda, oracle_lib, w, h, n):
    import oracle as O
    import torch
    rng = np.random.default_rng([w, h, n])
    cov = np.zeros((n, h, w), np.uint8)
    for i in range(n):
        cov[i][:, (i * w // n + np.arange(w // 2 + 1)) % w] = 255
    best = np.where(cov > 0, rng.random((n, h, w)), -1).argmax(0)
    seams = np.stack([((best == i) & (cov.max(0) > 0)).astype(np.uint8) * 255 for i in range(n)])
    imgs = rng.integers(0, 256, (n, h, w, 4)).astype(np.int16)
    imgs[..., 3] = 0
    imgs[cov == 0] = 0
    b = P.CudaTilingMultibandBlendFast()
    assert b.prepare(list(cov), list(seams), 16, 1)
    ref = O.Blender(cov, seams, 16, 1).blend(list(imgs))
    dev = [torch.from_numpy(i).cuda() for i in imgs]
    out = torch.zeros((h, w, 4), dtype=torch.uint8, device="cuda")
    b.blend(dev, out)
    assert np.array_equal(out.cpu().numpy()[..., :3], ref[..., :3])


@pytest.mark.parametrize("dst,levels,n", [(8, 3, 2), (36, 6, 3), (132, 7, 10), (260, 8, 5)])
@pytest.mark.parametrize("shape", [{}, {"tail_half_tiles": 0}, {"tail_cluster": 8, "tail_max_items": 64},
                                   {"tail_max_items": 1 << 20}, {"tail_max_items": 0, "small_blend_max_items": 1 << 20}],
                         ids=lambda s: ",".join(f"{k}={v}" for k, v in s.items()) or "default")
def test_render_levels_match_the_oracle(cuda, oracle_lib, dst, levels, n, shape):
    from _util import Prepared
    from panostitcher_gb300 import synth as S
    cams = [S.photo_param(0, 110.0, 360.0 * k / n, 25.0 * (k % 3) - 25.0) for k in range(n)]
    p = Prepared(S.RigConfig("tail", cams, (40, 30), (dst, dst // 2), levels, (0.8, 1.2)))
    p.r.set_launch_shape(**shape)
    for k in (0, 1):
        f = p.frames.frame(k)
        assert np.array_equal(p.product_render(f, p.luts)[..., :3], p.oracle_render(f, p.luts)[..., :3])
