"""Decoder frames of one call with and without aligned planes, in any order: one unaligned plane decides the conversion
of all.  Against the oracle."""
import numpy as np
import pytest

import panostitcher_gb300 as P
from panostitcher_gb300 import synth as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shifts", [(0, 0, 0, 0, 0, 0), (0, 0, 1, 0, 0, 0), (3, 0, 0, 8, 0, 1), (1, 2, 3, 4, 5, 6)])
@pytest.mark.parametrize("fmt", ["nv12", "yuv420p"])
def test_aligned_and_unaligned_frames(cuda, oracle_lib, fmt, shifts):
    import oracle as O
    import torch
    from _util import Prepared
    code, ofmt = (P.PS_FMT_NV12, O.FMT_NV12) if fmt == "nv12" else (P.PS_FMT_YUV420P, O.FMT_YUV420P)
    p = Prepared(S.scaled_rig(S.rig("c2"), 5))  # 384x216 frames
    w, h = p.cfg.src_size
    assert w % 8 == 0 and len(p.cfg.cams) == len(shifts)
    rng = np.random.default_rng(list(shifts))
    shapes = [(h, w), (h // 2, w)] if fmt == "nv12" else [(h, w), (h // 2, w // 2), (h // 2, w // 2)]
    frames, host = [], []
    for s in shifts:
        planes = [rng.integers(0, 256, q, dtype=np.uint8) for q in shapes]
        dev = []
        for q in planes:
            store = torch.zeros(q.size + 16, dtype=torch.uint8, device="cuda")
            store[s:s + q.size] = torch.from_numpy(q.ravel()).cuda()
            dev.append(store[s:s + q.size].view(q.shape))
        host.append(O.yuv_to_bgr32(planes, ofmt))
        frames.append(dev)
    ref = p.oracle_render(host, p.luts)
    out = torch.zeros((*p.cfg.dst_size[::-1], 4), dtype=torch.uint8, device="cuda")
    p.r.render_planar(frames, out, p.luts, code, check=True)
    assert np.array_equal(out.cpu().numpy()[..., :3], ref[..., :3])
