"""The fixed-point bilinear of the remap kernels.

CPU: the weights as the kernels form them (fp32 fma at 2^-24, the fourth the
rest of 2^24) keep a channel's sum within 2^-13 of the exact one, the
distance below which a pixel is recomputed exactly; the 64-bit recompute
rounds as the reference's double sequence wherever its sum is farther than
2^-40 from a tie.

GPU: every form a source can take (BGR32 and BGR24 at any alignment and
pitch, frames of one column or row, which take the general kernel) and maps
with exact rounding ties, last columns and rows, coordinates below 1 and
invalid values, against the oracle; no tolerance, the bytes are equal.
"""
import numpy as np
import pytest

import panostitcher_gb300 as P
from panostitcher_gb300 import synth as S


def _coords(rng, n):
    """Float map coordinates of every magnitude a frame has, with the fractions that matter."""
    whole = np.floor(rng.uniform(0, 2 ** rng.uniform(0, 13, n)))
    frac = rng.choice([0.0, 0.5, 0.25, 2.0 ** -12, 1 - 2.0 ** -12, -1.0], n)
    frac = np.where(frac < 0, rng.uniform(0, 1, n), frac)
    return (whole + frac).astype(np.float32)


def _fraction(m):
    return (m - np.floor(m)).astype(np.float32)  # exact in fp32


def _fixed_weight(a, b):
    """2 * bits(fma(a, b, 1)) - 0x7F000000: the product and sum are exact in double for these inputs, then one
    fp32 rounding."""
    t = (a.astype(np.float64) * b.astype(np.float64) + 1.0).astype(np.float32)
    return (2 * t.view(np.uint32).astype(np.int64) - 0x7F000000)


def test_fixed_point_sum_stays_within_the_near_tie_distance():
    rng = np.random.default_rng(11)
    n = 400_000
    x, y = _coords(rng, n), _coords(rng, n)
    small = rng.random(n) < 0.1  # coordinates below 1 with long fractions
    x[small] = rng.uniform(0, 1, small.sum()).astype(np.float32) ** 3
    fx, fy = _fraction(x), _fraction(y)
    gx, gy = (np.float32(1) - fx).astype(np.float32), (np.float32(1) - fy).astype(np.float32)
    w01, w10, w11 = _fixed_weight(fx, gy), _fixed_weight(gx, fy), _fixed_weight(fx, fy)
    w00 = (1 << 24) - w01 - w10 - w11
    p = rng.integers(0, 256, (4, n))
    p[:, : n // 2] = rng.choice([0, 255], (4, n // 2))  # the largest differences
    got = p[0] * w00 + p[1] * w01 + p[2] * w10 + p[3] * w11
    dx, dy = fx.astype(np.float64), fy.astype(np.float64)
    exact = (p[0] * (1 - dx) * (1 - dy) + p[1] * dx * (1 - dy) + p[2] * (1 - dx) * dy + p[3] * dx * dy) * 2.0 ** 24
    assert np.abs(got - exact).max() < 255 * 4 + 1  # 6.1e-5 of a grey level, half the near-tie distance
    assert 255 * 4 + 1 < 2048
    assert got.min() > -(1 << 23) and got.max() < (1 << 32) - (1 << 23)  # the rounded sum fits 32 bits


def test_integer_recompute_rounds_as_the_double_sequence():
    rng = np.random.default_rng(12)
    n = 200_000
    x, y = _coords(rng, n) + 1, _coords(rng, n) + 1
    x, y = x.astype(np.float32), y.astype(np.float32)
    fx, fy = _fraction(x).astype(np.float64), _fraction(y).astype(np.float64)
    ix, iy = fx * 2.0 ** 23, fy * 2.0 ** 23
    assert np.array_equal(ix, np.rint(ix)) and np.array_equal(iy, np.rint(iy))  # at most 23 fraction bits
    p = rng.integers(0, 256, (4, n))
    r = p[0] * ((1 - fx) * (1 - fy))  # the reference's order, each product and sum one IEEE rounding
    r = r + p[1] * (fx * (1 - fy))
    r = r + p[2] * ((1 - fx) * fy)
    r = r + p[3] * (fx * fy)
    one = 1 << 23
    jx, jy = ix.astype(np.int64), iy.astype(np.int64)
    total = (p[0] * ((one - jx) * (one - jy)) + p[1] * (jx * (one - jy)) + p[2] * ((one - jx) * jy) +
             p[3] * (jx * jy) + (1 << 45))
    frac = total & ((1 << 46) - 1)
    far = (frac > 64) & (frac < (1 << 46) - 64)
    assert np.array_equal((total >> 46)[far], np.rint(r)[far].astype(np.int64))
    assert far.mean() > 0.5 and not far.all()  # both branches occur


def _source(rng, h, w, fmt, pad, shift):
    """A (h, w, 3|4) CUDA image whose rows start `shift` bytes past an aligned address, `pad` bytes apart."""
    import torch
    c = 4 if fmt == "bgr32" else 3
    host = rng.integers(0, 256, (h, w, c), dtype=np.uint8)
    host[rng.random((h, w)) < 0.3] = rng.choice([0, 255])
    pitch = w * c + pad
    store = torch.zeros(shift + h * pitch, dtype=torch.uint8, device="cuda")
    t = store.as_strided((h, w, c), (pitch, c, 1), shift)
    t.copy_(torch.from_numpy(host))
    return host, t


def _maps(rng, H, W, sw, sh):
    def axis(n):
        v = rng.uniform(0, n, (H, W)).astype(np.float32)
        pick = rng.random((H, W))
        v = np.where(pick < 0.3, np.floor(v) + 0.5, v)          # exact ties
        v = np.where((pick > 0.3) & (pick < 0.4), n - 1 + v % 1, v)  # the last column or row
        v = np.where((pick > 0.4) & (pick < 0.45), v % 1, v)    # below 1
        v = np.where((pick > 0.45) & (pick < 0.5), rng.choice([0.0, -0.0, n, -1.0, np.nan, np.inf, -1e-9, -1e30]), v)
        return np.minimum(v, np.nextafter(np.float32(n), np.float32(0)), where=pick < 0.45, out=v.astype(np.float32))
    return axis(sw).astype(np.float32), axis(sh).astype(np.float32)


@pytest.mark.gpu
@pytest.mark.parametrize("sw,sh", [(1, 7), (9, 1), (2, 2), (3, 5), (33, 17), (200, 120)])
@pytest.mark.parametrize("fmt,pad,shift", [("bgr32", 0, 0), ("bgr32", 12, 4), ("bgr24", 0, 0), ("bgr24", 1, 1),
                                           ("bgr24", 2, 3), ("bgr24", 3, 2)])
def test_reproject_of_every_source_form(cuda, oracle_lib, sw, sh, fmt, pad, shift):
    import oracle as O
    import torch
    from panostitcher_gb300.render import reproject_to_16s
    rng = np.random.default_rng([sw, sh, pad, shift])
    host, dev = _source(rng, sh, sw, fmt, pad, shift)
    lut = rng.integers(0, 256, (3, 256), dtype=np.uint8)
    for W, H in ((1, 1), (15, 2), (17, 3), (64, 16), (131, 35)):
        xm, ym = _maps(rng, H, W, sw, sh)
        dst = torch.full((H, W, 4), 7, dtype=torch.int16, device="cuda")
        for table in (lut, None):
            reproject_to_16s(dev, torch.from_numpy(xm).cuda(), torch.from_numpy(ym).cuda(), dst,
                             None if table is None else torch.from_numpy(table).cuda())
            ref = O.reproject_16s(host, xm, ym, table)
            assert np.array_equal(dst.cpu().numpy()[..., :3], ref[..., :3]), (W, H)


@pytest.mark.gpu
@pytest.mark.parametrize("src", [(1, 8), (8, 1), (2, 2), (37, 23)])
def test_render_of_small_and_unaligned_sources(cuda, oracle_lib, src):
    from _util import Prepared
    import torch
    cams = [S.photo_param(1, 200.0, 0.0), S.photo_param(1, 200.0, 180.0)]
    cfg = S.RigConfig("small", cams, src, (132, 66), 4, (0.8, 1.2))
    p = Prepared(cfg)
    rng = np.random.default_rng(src)
    for fmt, pad, shift in (("bgr32", 4, 8), ("bgr24", 1, 1), ("bgr24", 2, 3)):
        pairs = [_source(rng, src[1], src[0], fmt, pad, shift) for _ in cams]
        out = torch.zeros((66, 132, 4), dtype=torch.uint8, device="cuda")
        p.r.render([d for _, d in pairs], out, p.luts, check=True)
        ref = p.oracle_render([h for h, _ in pairs], p.luts)
        assert np.array_equal(out.cpu().numpy()[..., :3], ref[..., :3]), fmt


@pytest.mark.gpu
@pytest.mark.parametrize("n", [2, 9])
def test_linear_render_takes_every_format_alike(cuda, oracle_lib, n):
    import torch
    cams = [S.photo_param(0, 100.0, 360.0 * k / n, 20.0 * (k % 3) - 20.0) for k in range(n)]
    cfg = S.RigConfig("lin", cams, (61, 47), (196, 98), 4, (0.8, 1.2))
    r = P.CudaPanoramaRender2()
    r.prepare(cams, 0, 9, cfg.src_size, cfg.dst_size, check=True)
    luts = S.luts(cfg)
    frames = S.FrameSource(cfg).frame(0)
    maps = [r.maps(i, cfg.dst_size) for i in range(n)]
    wts = np.stack([r.linear_weight(i, cfg.dst_size) for i in range(n)])
    import oracle as O
    ref = O.linear_render(frames, luts, [m[0] for m in maps], [m[1] for m in maps], wts)
    for dev in ([torch.from_numpy(f).cuda() for f in frames],
                [torch.from_numpy(np.ascontiguousarray(f[..., :3])).cuda() for f in frames]):
        out = torch.zeros((98, 196, 4), dtype=torch.uint8, device="cuda")
        r.render(dev, out, luts, check=True)
        assert np.array_equal(out.cpu().numpy()[..., :3], ref[..., :3])
