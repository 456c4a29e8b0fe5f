"""What the launch shape's values mean: small_blend_max_items hands k_blend_small the levels of at most that many tiles
(0 none, 128 the default), and the two values that choose no launch change nothing and wait for nothing."""
import numpy as np
import pytest

import panostitcher_gb300 as P
from panostitcher_gb300 import synth as S

pytestmark = pytest.mark.gpu


@pytest.fixture
def rig(cuda):
    import torch
    cfg = S.scaled_rig(S.rig("c2"), 8)  # 512x256
    r = P.CudaPanoramaRender2()
    r.prepare(cfg.cams, 1, cfg.levels, cfg.src_size, cfg.dst_size, check=True)
    rng = np.random.default_rng(4)
    src = [torch.from_numpy(rng.integers(0, 256, (*cfg.src_size[::-1], 4), dtype=np.uint8)).cuda() for _ in cfg.cams]
    return r, src, torch.zeros((*cfg.dst_size[::-1], 4), dtype=torch.uint8, device="cuda"), cfg


def _small_launches(rig):
    r, src, dst, _ = rig
    r.profile(True)
    before = r.profile_read(6)[0]
    r.render(src, dst, None, check=True)
    n = r.profile_read(6)[0] - before
    r.profile(False)
    return n, dst.cpu()


def test_small_blend_max_items(rig):
    r, _, _, cfg = rig
    assert r.launch_shape() == P.CudaPanoramaRender2.SHAPE_DEFAULT
    w, h = cfg.dst_size
    tiles = []  # of the levels above 0
    for _ in range(r.num_levels):
        w, h = (w + 1) // 2, (h + 1) // 2
        tiles.append(-(-w // 64) * -(-h // 16))
    want = None
    r.set_launch_shape(tail_max_items=0)
    for most in (128, 0, 1, 2, tiles[0] - 1, tiles[0]):
        r.set_launch_shape(small_blend_max_items=most)
        n, out = _small_launches(rig)
        assert n == sum(t <= most for t in tiles), most
        want = out if want is None else want
        assert (out == want).all()


def test_values_without_launches_wait_for_nothing(rig):
    import torch
    r, src, dst, _ = rig
    s = torch.cuda.Stream()
    for _ in range(9):  # every state slot has its launches recorded
        r.render(src, dst, None, stream=s, check=True)
    torch.cuda.synchronize()
    want = dst.cpu()
    dst.zero_()
    torch.cuda.synchronize()
    done = torch.cuda.Event()
    with torch.cuda.stream(s):
        torch.cuda._sleep(2_000_000_000)  # a second
    r.render(src, dst, None, stream=s, check=True)
    done.record(s)
    r.set_launch_shape(tail_half_tiles=0, remap_defer_ties=0)
    assert not done.query()
    shape = r.launch_shape()
    assert shape["tail_half_tiles"] == 0 and shape["remap_defer_ties"] == 0
    r.render(src, dst, None, stream=s, check=True)
    assert not done.query()
    torch.cuda.synchronize()
    assert (dst.cpu() == want).all()
