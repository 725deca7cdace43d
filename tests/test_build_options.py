"""The schedule rules of the runtime (tile depth, stretches of the line sweeps) count the CTAs per SM
that the kernels are compiled for: a build option that changes the one changes the other.  A
host program over the runtime's own header, compiled with and without the options; no GPU."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
NVCC = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"

PROGRAM = """
#include <cstdio>
#include "gdfv_launch.h"
using namespace gdfv;
int main() {
    std::printf("%d %d %d %d %d %d\\n", tile_ctas_per_sm(0, false), tile_ctas_per_sm(0, true), tile_ctas_per_sm(1, false),
                tile_ctas_per_sm(1, true), sweep_ctas_per_sm(false), sweep_ctas_per_sm(true));
}
"""


@pytest.mark.skipif(not os.path.exists(NVCC), reason="no nvcc")
@pytest.mark.parametrize("options, want", [
    ([], [2, 1, 3, 2, 4, 2]),
    (["GDFV_MINB_FP64=3", "GDFV_MINB_FP32=4", "GDFV_MINB_MHD_FP32=1", "GDFV_MARCH_MINB=5", "GDFV_MARCH_MINB_MHD=3"],
     [3, 1, 4, 1, 5, 3]),
])
def test_residency_follows_the_build_options(tmp_path, options, want):
    src, exe = tmp_path / "options.cu", tmp_path / "options"
    src.write_text(PROGRAM)
    subprocess.run([NVCC, "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a", "--expt-relaxed-constexpr",
                    "-I", os.path.join(ROOT, "gdtk-rmhd_b200", "csrc"), "-I", os.path.join(ROOT, "include"),
                    *("-D" + o for o in options), "-o", str(exe), str(src)], check=True, capture_output=True)
    out = subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout
    assert [int(v) for v in out.split()] == want
