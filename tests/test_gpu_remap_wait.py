"""The remap's own bounded waits: the probe's wait runs out in k_remap too, in every build of it, the check names the
remap, and the render carries on.  The blender has no remap and names none."""
import numpy as np
import pytest

import panostitcher_gb300 as P
from panostitcher_gb300 import synth as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("source", ["bgr32", "bgr24", "map-free"])
def test_probe_reaches_the_remap(cuda, source):
    import torch
    cfg = S.scaled_rig(S.rig("c2"), 8)
    r = P.CudaPanoramaRender2()
    r.set_map_free(source == "map-free")
    r.prepare(cfg.cams, 1, cfg.levels, cfg.src_size, cfg.dst_size, check=True)
    rng = np.random.default_rng(3)
    c = 3 if source == "bgr24" else 4
    src = [torch.from_numpy(rng.integers(0, 256, (*cfg.src_size[::-1], c), dtype=np.uint8)).cuda() for _ in cfg.cams]
    outs = [torch.zeros((*cfg.dst_size[::-1], 4), dtype=torch.uint8, device="cuda") for _ in range(3)]
    r.render(src, outs[0], None, check=True)
    r.set_wait_probe(1000)
    r.render(src, outs[1], None, check=True)
    assert not r.check_status(check=False)
    assert "bounded wait of the remap and of a blend kernel" in r.last_error
    r.set_wait_probe(0)
    r.render(src, outs[2], None, check=True)
    assert r.check_status()
    assert torch.equal(outs[0], outs[1]) and torch.equal(outs[0], outs[2])  # a wait beside the ring changes nothing


def test_blender_names_the_blend_alone(cuda):
    import torch
    b = P.CudaTilingMultibandBlendFast()
    m = np.full((64, 128), 255, np.uint8)
    assert b.prepare([m], [m], 3)
    b.set_wait_probe(1000)
    b.blend([torch.zeros((64, 128, 4), dtype=torch.int16, device="cuda")], torch.zeros((64, 128, 4), dtype=torch.uint8, device="cuda"))
    assert b.check_status() == P._lib.PS_ETIMEOUT
    text = P._lib.lib().ps_last_error().decode()
    assert "a blend kernel" in text and "remap" not in text
