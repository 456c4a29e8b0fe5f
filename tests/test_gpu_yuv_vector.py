"""The eight-pixel conversions and the per-block ones beside them: widths, pitches and plane addresses on both
sides of the rule that chooses, against the oracle."""
import numpy as np
import pytest

import panostitcher_gb300 as P

pytestmark = pytest.mark.gpu


def _plane(host, pad, shift):
    import torch
    h, w = host.shape[:2]
    c = host.shape[2] if host.ndim == 3 else 1
    store = torch.zeros(shift + h * (w * c + pad), dtype=torch.uint8, device="cuda")
    size, stride = ((h, w, c), (w * c + pad, c, 1)) if host.ndim == 3 else ((h, w), (w + pad, 1))
    t = store.as_strided(size, stride, shift)
    t.copy_(torch.from_numpy(host))
    return t


@pytest.mark.parametrize("w,h", [(8, 2), (16, 6), (10, 4), (1032, 18), (1024, 2), (1026, 10)])
@pytest.mark.parametrize("fmt", ["nv12", "yuv420p"])
@pytest.mark.parametrize("pad,shift", [(0, 0), (16, 0), (8, 16), (4, 4), (0, 8), (2, 1)])
def test_conversions_match_the_oracle(cuda, oracle_lib, w, h, fmt, pad, shift):
    import oracle as O
    from panostitcher_gb300.render import cvt_bgr32_to_yuv, cvt_yuv_to_bgr32
    rng = np.random.default_rng([w, h, pad, shift])
    code, ofmt = (P.PS_FMT_NV12, O.FMT_NV12) if fmt == "nv12" else (P.PS_FMT_YUV420P, O.FMT_YUV420P)
    bgr = rng.integers(0, 256, (h, w, 4), dtype=np.uint8)
    bgr[..., 3] = 0
    bgr[0, :2] = 255
    img = _plane(bgr, pad // 4 * 4, shift // 4 * 4)  # BGR32 images are 4-byte aligned
    want = O.bgr32_to_yuv(bgr, ofmt)
    planes = [_plane(np.zeros_like(p), pad, shift) for p in want]
    cvt_bgr32_to_yuv(img, planes, code)
    for a, b in zip(planes, want):
        assert np.array_equal(a.cpu().numpy(), b)
    src = [rng.integers(0, 256, p.shape, dtype=np.uint8) for p in want]
    out = _plane(np.full((h, w, 4), 9, np.uint8), pad // 4 * 4, shift // 4 * 4)
    cvt_yuv_to_bgr32([_plane(p, pad, shift) for p in src], out, code)
    assert np.array_equal(out.cpu().numpy(), O.yuv_to_bgr32(src, ofmt))
