"""A render on a stream that is being captured: with device buffers alone the kernels would go to that stream, so the run
looks first.  The call is refused, whatever the capture's mode, nothing of it runs, and the render works as before on
every state slot afterwards.  In a process of its own: a capture that fails leaves its mark on the framework that
began it."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SCRIPT = r"""
import sys
sys.path[:0] = [ROOT, ROOT + "/tests"]
import numpy as np
import torch
from panostitcher_gb300 import synth as S
from _util import Prepared
torch.cuda.set_device(0)
p = Prepared(S.scaled_rig(S.rig("c1"), 8))
f = p.frames.frame(0)
ref = torch.from_numpy(p.oracle_render(f, p.luts)[..., :3])
dev = [torch.from_numpy(x).cuda() for x in f]
dst = torch.zeros((*p.cfg.dst_size[::-1], 4), dtype=torch.uint8, device="cuda")
s = torch.cuda.Stream()
for _ in range(WARM):
    p.r.render(dev, dst, p.luts, stream=s, check=True)
torch.cuda.synchronize()
dst.fill_(7)
torch.cuda.synchronize()
g = torch.cuda.CUDAGraph()
with torch.cuda.stream(s):
    g.capture_begin(capture_error_mode=MODE)
    ok = p.r.render(dev, dst, p.luts, stream=s, check=False)
    text = p.r.last_error
    try:
        g.capture_end()
    except Exception:
        pass
assert not ok and "captur" in text, text
torch.cuda.synchronize()
assert bool((dst == 7).all())
for k in range(10):  # all state slots, on both streams
    dst.fill_(9)
    torch.cuda.synchronize()
    p.r.render(dev, dst, p.luts, stream=s if k % 2 else None, check=True)
    torch.cuda.synchronize()
    assert torch.equal(dst[..., :3].cpu(), ref), k
print("done")
"""


@pytest.mark.parametrize("mode", ["global", "thread_local", "relaxed"])
@pytest.mark.parametrize("warm", [0, 9])
def test_render_on_a_capturing_stream_is_refused(cuda, oracle_lib, mode, warm):
    code = SCRIPT.replace("ROOT", repr(ROOT)).replace("MODE", repr(mode)).replace("WARM", str(warm))
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=240)
    assert r.returncode == 0 and r.stdout.endswith("done\n"), r.stdout + r.stderr
