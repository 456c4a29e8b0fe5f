"""Decoder planes to BGR32 images at every placement that the entry point accepts: base addresses on a multiple of 4,
8 or 16 bytes with row pitches that are or are not multiples of 8, against the oracle."""
import numpy as np
import pytest

import panostitcher_gb300 as P

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h", [(2, 2), (8, 4), (10, 4), (1024, 6), (1026, 6)])
@pytest.mark.parametrize("fmt", ["nv12", "yuv420p"])
@pytest.mark.parametrize("shift", [0, 4, 8, 12, 16])
@pytest.mark.parametrize("pad", [0, 4, 8, 16])
def test_planes_to_bgr32(cuda, oracle_lib, w, h, fmt, shift, pad):
    import oracle as O
    import torch
    from panostitcher_gb300.render import cvt_yuv_to_bgr32
    rng = np.random.default_rng([w, h, shift, pad])
    code, ofmt = (P.PS_FMT_NV12, O.FMT_NV12) if fmt == "nv12" else (P.PS_FMT_YUV420P, O.FMT_YUV420P)
    shapes = [(h, w), (h // 2, w)] if fmt == "nv12" else [(h, w), (h // 2, w // 2), (h // 2, w // 2)]
    src = [rng.integers(0, 256, s, dtype=np.uint8) for s in shapes]
    pitch = 4 * w + pad
    store = torch.full((shift + h * pitch + 16,), 9, dtype=torch.uint8, device="cuda")
    out = store.as_strided((h, w, 4), (pitch, 4, 1), shift)
    assert out.data_ptr() % 16 == shift % 16
    want = store.cpu().numpy()
    np.lib.stride_tricks.as_strided(want[shift:], (h, w, 4), (pitch, 4, 1))[:] = O.yuv_to_bgr32(src, ofmt)
    cvt_yuv_to_bgr32([torch.from_numpy(p).cuda() for p in src], out, code)
    assert np.array_equal(store.cpu().numpy(), want)  # and nothing beside the image
