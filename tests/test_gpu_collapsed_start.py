"""The collapsed levels before any frame: zeros on every level, after a refused frame too and again after a new prepare;
a state slot that a refused frame took leaves the next frames as they are."""
import numpy as np
import pytest

import panostitcher_gb300 as P
from panostitcher_gb300 import synth as S

pytestmark = pytest.mark.gpu


def test_levels_are_zero_before_the_first_frame(cuda, oracle_lib):
    import torch
    from _util import Prepared
    p = Prepared(S.scaled_rig(S.rig("c2"), 8))
    sizes = p.ob.sizes

    def zeros():
        return all(not p.r.collapsed(j, sizes[j]).any() for j in range(1, p.r.num_levels + 1))

    assert p.r.num_levels > 3 and zeros()
    f = p.frames.frame(0)
    with pytest.raises(P.PsError):
        p.r.render(f[:-1], np.zeros((*p.cfg.dst_size[::-1], 4), np.uint8), p.luts, check=True)
    assert zeros()
    ref = p.oracle_render(f, p.luts)
    assert np.array_equal(p.product_render(f, p.luts)[..., :3], ref[..., :3])
    torch.cuda.synchronize()
    assert not zeros()
    p.r.prepare(p.cfg.cams, 1, p.cfg.levels, p.cfg.src_size, p.cfg.dst_size, check=True)
    assert zeros()
