"""Uniform tiles (one camera at weight 256) whose collapsed footprint leaves the packed range -256..767, in k_blend and
k_blend_rows, so that their general path takes them.  A collapsed value is a linear function of the images up to
rounding; every pixel black or white by the sign of its coefficient gives the largest and the smallest there is.
Seams in rings around the tile let another camera decide every level, whose Laplacians then add up."""
import numpy as np
import pytest

import panostitcher_gb300 as P

pytestmark = pytest.mark.gpu

LOW, HIGH = -256, 767  # what the packed path holds


def _rings(w, h, cx, cy, a, b):
    """Seams: a rectangle of half sizes a x b around (cx, cy), rings around it, the rest."""
    y, x = np.mgrid[0:h, 0:w]
    seams, inner, s = [], np.zeros((h, w), bool), 1.0
    while b * s < h / 2:
        m = ((np.abs(x + 0.5 - cx) < a * s ** 0.6) & (np.abs(y + 0.5 - cy) < b * s)) | inner
        seams.append(m & ~inner)
        inner, s = m, 2 * s
    seams.append(~inner)
    return np.stack(seams).astype(np.uint8) * 255


def _coefficients(seams, levels, level, x, y):
    """Of collapsed pixel (x, y) of `level`, by the images' pixels (borders only roughly)."""
    import torch
    import torch.nn.functional as F
    k = torch.tensor([1.0, 4, 6, 4, 1]) / 16
    k = (k[:, None] * k)[None, None]

    def pad(t):
        return F.pad(F.pad(t, (2, 2, 0, 0), mode="circular"), (0, 0, 2, 2), mode="replicate")

    def down(t):
        return F.conv2d(pad(t), k, stride=2)

    def up(t):
        z = torch.zeros(t.shape[0], 1, 2 * t.shape[2], 2 * t.shape[3])
        z[:, :, ::2, ::2] = t
        return F.conv2d(pad(z), 4 * k)

    img = torch.zeros((len(seams), 1, *seams.shape[1:]), requires_grad=True)
    G, W = [img], [torch.from_numpy(seams / 255.0).float()[:, None]]
    for _ in range(levels):
        G.append(down(G[-1]))
        W.append(down(W[-1]))
    C = None
    for j in range(levels, level - 1, -1):
        N = ((G[j] if j == levels else G[j] - up(G[j + 1])) * W[j]).sum(0, keepdim=True)
        C = N if C is None else N + up(C)
    C[0, 0, y, x].backward()
    return img.grad[:, 0].numpy()


# level 0 in k_blend_rows and in k_blend (2560 tiles), level 1 in k_blend_rows (one level less to add up: low only)
@pytest.mark.parametrize("w,h,j", [(1536, 1024, 0), (2560, 1024, 0), (2048, 1024, 1)])
def test_collapsed_values_beyond_the_packed_range(cuda, oracle_lib, w, h, j):
    import oracle as O
    import torch
    levels, s = 9, 1 << j
    tx, ty = w // 2 // (64 * s), h // 2 // (16 * s)  # the uniform tile
    cx, cy = (tx * 64 + 32) * s, (ty * 16 + 8) * s
    seams = _rings(w, h, cx, cy, 32 * s + 4 * j, 8 * s + 4 * j)
    n = len(seams)
    g = _coefficients(seams, levels, j + 1, cx // (2 * s), cy // (2 * s))
    rng = np.random.default_rng([w, h, j])
    noise = rng.integers(0, 256, (n, h, w))
    imgs = np.zeros((n, h, w, 4), np.int16)
    imgs[..., 0] = np.where(g == 0, noise, (g < 0) * 255)
    imgs[..., 1] = np.where(g == 0, 255 - noise, (g > 0) * 255)
    imgs[..., 2] = noise
    cov = np.full((n, h, w), 255, np.uint8)
    ob = O.Blender(cov, seams, levels)
    assert ob.levels == levels
    assert (ob.weight(0, j)[ty * 16:ty * 16 + 16, tx * 64:tx * 64 + 64] == 256).all()  # a uniform tile
    ref, _, collapsed = ob.blend(list(imgs), pyramids=True)
    c = collapsed[j + 1][ty * 8 - 1:ty * 8 + 9, tx * 32 - 1:tx * 32 + 33]  # its footprint
    assert c[..., 0].min() < LOW and (c[..., 1].max() > HIGH or j), (c[..., 0].min(), c[..., 1].max())
    b = P.CudaTilingMultibandBlendFast()
    assert b.prepare(list(cov), list(seams), levels, 2), b.last_error
    dev = [torch.from_numpy(i).cuda() for i in imgs]
    for ch in (4, 3):
        out = torch.full((h, w, ch), 7, dtype=torch.uint8, device="cuda")
        b.blend(dev, out)
        assert np.array_equal(out.cpu().numpy()[..., :3], ref[..., :3])
