"""The tail's cluster width and the other one that the autotuner times: never the width in use under another value."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SOURCE = """
#include "ps_internal.h"
#include <cstdio>
int main()
{
    for (int widest : {8, 16})
        for (int cams = 1; cams <= 64; cams++)
            for (int asked : {0, 8, 16})
                std::printf("%d %d %d %d %d\\n", widest, cams, asked, ps::tailClusterWidth(asked, cams, widest),
                            ps::tailClusterOther(asked, cams, widest));
}
"""


def test_the_other_width_is_another(tmp_path):
    cuda = os.path.join(os.path.dirname(os.path.dirname(shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc")), "include")
    if not os.path.isdir(cuda):
        pytest.skip("no CUDA headers")
    (tmp_path / "t.cpp").write_text(SOURCE)
    subprocess.check_call(["g++", "-std=c++17", "-I" + os.path.join(ROOT, "panostitcher_gb300", "csrc"),
                           "-I" + os.path.join(ROOT, "include"), "-I" + cuda, str(tmp_path / "t.cpp"), "-o",
                           str(tmp_path / "t")])
    rows = [tuple(map(int, r.split())) for r in subprocess.check_output([str(tmp_path / "t")], text=True).splitlines()]
    width = {r[:3]: r[3] for r in rows}
    for widest, cams, asked, w, other in rows:
        assert w == min(widest, asked or (8 if cams <= 8 else 16))
        if widest == 8:
            assert other == 0  # nothing else to time
        else:
            assert other in (8, 16) and width[widest, cams, other] == other != w
