"""k_tail, which runs every level of at most 32x16 pixels of up to 16 cameras: the sizes where its first level lies
at or beside that limit, its camera limits (a CTA a camera, two a CTA, one more than it takes), cameras that cover
nothing.  The collapsed levels are the oracle's bytes through the blend; equal integers, so no tolerance."""
import numpy as np
import pytest

import panostitcher_gb300 as P

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 8, 12, 16, 17])
@pytest.mark.parametrize("w,h", [(32, 16), (64, 32), (65, 32), (62, 33), (40, 130), (257, 9)])
def test_blend_matches_the_oracle(cuda, oracle_lib, w, h, n):
    import oracle as O
    import torch
    rng = np.random.default_rng([w, h, n])
    cov = np.zeros((n, h, w), np.uint8)
    for i in range(n):
        if n > 2 and i % 5 == 3:
            continue  # a camera that covers nothing
        cov[i][:, (i * w // n + np.arange(max(1, w // 3))) % w] = 255
    best = np.where(cov > 0, rng.random((n, h, w)), -1).argmax(0)
    seams = np.stack([((best == i) & (cov.max(0) > 0)).astype(np.uint8) * 255 for i in range(n)])
    imgs = rng.integers(0, 256, (n, h, w, 4)).astype(np.int16)
    imgs[..., 3] = 0
    imgs[cov == 0] = 0
    b = P.CudaTilingMultibandBlendFast()
    assert b.prepare(list(cov), list(seams), 16, 1), b.last_error
    ref = O.Blender(cov, seams, 16, 1).blend(list(imgs))
    out = torch.zeros((h, w, 4), dtype=torch.uint8, device="cuda")
    for _ in range(2):
        b.blend([torch.from_numpy(i).cuda() for i in imgs], out)
        assert np.array_equal(out.cpu().numpy()[..., :3], ref[..., :3])


@pytest.mark.parametrize("n", [7, 13])
@pytest.mark.parametrize("cluster", [0, 8, 16])
@pytest.mark.parametrize("tail", [1, 16])
def test_cluster_widths(cuda, oracle_lib, n, cluster, tail):
    from _util import Prepared
    from panostitcher_gb300 import synth as S
    cams = [S.photo_param(0, 100.0, 360.0 * k / n, 20.0 * (k % 3) - 20.0) for k in range(n)]
    p = Prepared(S.RigConfig("tail", cams, (40, 30), (140, 70), 7, (0.8, 1.2)))
    p.r.set_launch_shape(tail_cluster=cluster, tail_max_items=tail)
    f = p.frames.frame(0)
    assert np.array_equal(p.product_render(f, p.luts)[..., :3], p.oracle_render(f, p.luts)[..., :3])
