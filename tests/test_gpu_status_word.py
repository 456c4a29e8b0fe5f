"""A wait that ran out is reported by the next check, whatever is called in between: a refused image neither erases it
nor leaves anything behind itself."""
import numpy as np
import pytest

import panostitcher_gb300 as P
from panostitcher_gb300 import _lib as L

pytestmark = pytest.mark.gpu


def test_refused_image_keeps_the_timeout(cuda):
    import torch
    h, w = 128, 256
    b = P.CudaTilingMultibandBlendFast()
    cov = np.full((h, w), 255, np.uint8)
    cov[:, :5] = 0
    assert b.prepare([cov], [cov], 5)
    img = torch.zeros((h, w, 4), dtype=torch.int16, device="cuda")
    out = torch.zeros((h, w, 4), dtype=torch.uint8, device="cuda")
    outside, outsized = img.clone(), img.clone()
    outside[3, 2, 1] = 1
    outsized[7, 99, 0] = 256
    for bad in (outside, outsized):
        with pytest.raises(P.PsError):
            b.blend([bad], out)
        assert b.check_status() == L.PS_OK  # the refusal itself leaves nothing
        b.set_wait_probe(1000)
        b.blend([img], out)
        b.set_wait_probe(0)
        with pytest.raises(P.PsError):
            b.blend([bad], out)
        assert b.check_status() == L.PS_ETIMEOUT
        assert b.check_status() == L.PS_OK
