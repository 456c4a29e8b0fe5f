"""k_pyrdown's tiles where a warp's rows, the halo columns, the divisor-free path and the border's index maps meet: the
blend of their levels against the oracle's, as equal integers (no tolerance).  Level 0 is random; half of the
cameras cover everything (alpha 256 on every tile), the rest ragged parts."""
import numpy as np
import pytest

import panostitcher_gb300 as P

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h", [(64, 33), (67, 35), (130, 66), (133, 71), (198, 130), (260, 132), (324, 201), (641, 75)])
def test_levels_match_the_oracle(cuda, oracle_lib, w, h):
    import oracle as O
    import torch
    rng = np.random.default_rng([w, h])
    n = 4
    cov = np.full((n, h, w), 255, np.uint8)
    cov[1, :, w // 2 + 1:] = 0
    cov[2, h // 3:2 * h // 3 + 1] = 0
    cov[2][rng.random((h, w)) < 0.02] = 0
    best = np.where(cov > 0, rng.random((n, 1, 1)) + 0.2 * rng.random((n, h // 8 + 1, w // 8 + 1)).repeat(8, 1).repeat(8, 2)[:, :h, :w],
                    -1).argmax(0)
    seams = np.stack([(best == i).astype(np.uint8) * 255 for i in range(n)])
    imgs = rng.integers(0, 256, (n, h, w, 4)).astype(np.int16)
    imgs[0, :, :, :3] = 255  # the largest sums
    imgs[..., 3] = 0
    imgs[cov == 0] = 0
    b = P.CudaTilingMultibandBlendFast()
    assert b.prepare(list(cov), list(seams), 4, 1), b.last_error
    ref = O.Blender(cov, seams, 4, 1).blend(list(imgs))
    out = torch.zeros((h, w, 4), dtype=torch.uint8, device="cuda")
    b.blend([torch.from_numpy(i).cuda() for i in imgs], out)
    assert np.array_equal(out.cpu().numpy()[..., :3], ref[..., :3])
