"""Renders whose buffers are all on the device run on the caller's stream: their order with the caller's own
work, with renders that copy host buffers and with renders on other streams is what it was, and every frame is
the oracle's."""
import numpy as np
import pytest

import panostitcher_gb300 as P
from panostitcher_gb300 import synth as S

from _util import Prepared

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("slots", [1, 3, 8])
@pytest.mark.parametrize("default_stream", [True, False])
def test_device_and_host_frames_in_turn(cuda, oracle_lib, slots, default_stream):
    import torch
    cfg = S.scaled_rig(S.rig("c2"), 8)
    p = Prepared(cfg)
    p.r.set_frames_in_flight(slots)
    p.r.prepare(cfg.cams, 1, cfg.levels, cfg.src_size, cfg.dst_size, check=True)
    W, H = cfg.dst_size
    frames = [p.frames.frame(k) for k in range(4)]
    refs = [p.oracle_render(f, p.luts)[..., :3] for f in frames]
    stream = torch.cuda.current_stream() if default_stream else torch.cuda.Stream()
    handle = None if default_stream else stream
    staging = [torch.empty((cfg.src_size[1], cfg.src_size[0], 4), dtype=torch.uint8, device="cuda") for _ in cfg.cams]
    outs = []
    with torch.cuda.stream(stream):
        for k in range(20):
            f, kind = frames[k % 4], k % 3
            if kind == 2:  # host frames, host canvas: the render's own streams
                out = np.zeros((H, W, 4), np.uint8)
                p.r.render(f, out, p.luts, stream=handle, check=True)
            else:          # the caller's stream writes the one staging before each frame and copies the canvas after
                for s, h in zip(staging, f):
                    s.copy_(torch.from_numpy(h))
                dev = torch.zeros((H, W, 4), dtype=torch.uint8, device="cuda")
                src = f if kind == 1 else staging  # host frames with a device canvas go the other way again
                p.r.render(src, dev, p.luts, stream=handle, check=True)
                out = dev.clone()
                dev.fill_(7)
            outs.append((k % 4, out))
    torch.cuda.synchronize()
    for k, o in outs:
        o = o if isinstance(o, np.ndarray) else o.cpu().numpy()
        assert np.array_equal(o[..., :3], refs[k])


def test_streams_and_reprepare(cuda, oracle_lib):
    import torch
    cfg = S.scaled_rig(S.rig("c1"), 4)
    p = Prepared(cfg)
    W, H = cfg.dst_size
    frames = [[torch.from_numpy(x).cuda() for x in p.frames.frame(k)] for k in range(5)]
    refs = [p.oracle_render(p.frames.frame(k), p.luts)[..., :3] for k in range(5)]
    for _ in range(2):
        streams = [torch.cuda.Stream() for _ in range(5)]
        outs = [torch.zeros((H, W, 4), dtype=torch.uint8, device="cuda") for _ in range(20)]
        torch.cuda.synchronize()  # the buffers above were made on the default stream
        for k, o in enumerate(outs):
            p.r.render(frames[k % 5], o, p.luts, stream=streams[k % 5], check=True)
        # a new prepare and a change of shape wait for the frames on the callers' streams
        p.r.set_launch_shape(tail_max_items=0)
        p.r.set_launch_shape(**P.CudaPanoramaRender2.SHAPE_DEFAULT)
        p.r.prepare(cfg.cams, 1, cfg.levels, cfg.src_size, cfg.dst_size, check=True)
        torch.cuda.synchronize()
        for k, o in enumerate(outs):
            assert np.array_equal(o.cpu().numpy()[..., :3], refs[k % 5])
