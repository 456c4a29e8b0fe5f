"""k_linear over several rigs in one launch: segments that end inside a CTA's tiles (canvases of 1, 4, 25 and 121 tiles),
rigs of different camera counts, so that the tables in shared memory change on the way.  Equal bytes, no tolerance."""
import numpy as np
import pytest

import panostitcher_gb300 as P
from panostitcher_gb300 import synth as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("order", [(0, 1, 2, 3), (3, 0, 2, 1)])
def test_batch_of_linear_rigs(cuda, order):
    import torch
    rigs = []
    for dst, n in ((32, 2), (64, 5), (152, 3), (332, 7)):
        cams = [S.photo_param(0, 130.0, 360.0 * k / n) for k in range(n)]
        cfg = S.RigConfig("lin", cams, (60, 40), (dst, dst // 2), 2, (0.8, 1.2))
        r = P.CudaPanoramaRender2()
        r.prepare(cfg.cams, 0, 3, cfg.src_size, cfg.dst_size, check=True)
        frames = [torch.from_numpy(np.ascontiguousarray(f)).cuda() for f in S.FrameSource(cfg).frame(dst)]
        out = torch.zeros((dst // 2, dst, 4), dtype=torch.uint8, device="cuda")
        r.render(frames, out, S.luts(cfg), check=True)
        rigs.append((r, frames, S.luts(cfg), out))
    rigs = [rigs[k] for k in order]
    outs = [torch.full_like(x[3], 7) for x in rigs]
    P.render_batch([x[0] for x in rigs], [x[1] for x in rigs], outs, [x[2] for x in rigs])
    torch.cuda.synchronize()
    for x, out in zip(rigs, outs):
        assert torch.equal(out[..., :3], x[3][..., :3])
