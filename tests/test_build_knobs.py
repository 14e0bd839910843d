"""Build-time tile knobs keep the kernels' shared memory large enough."""
import subprocess

import pytest

from aapm_lowdosectimagerecon_competition_b200 import build

CODE = """
#include "ddfan_dd_kernels.cuh"
using namespace ddfan;
// the totals of the wide body's channels and of the thin body's two
template <int SV> constexpr bool holds() { return DdFwdTile<SV>::DYN >= (DDFAN_DD_FWD_CG > 2 ? DDFAN_DD_FWD_CG : 2) * SV * 256 * 4; }
static_assert(holds<1>() && holds<4>() && holds<8>(), "a forward thread's totals");
"""


@pytest.mark.parametrize("channels", [1, 2, 3])
def test_forward_totals_fit_for_every_channel_count(tmp_path, channels):
    src = tmp_path / "knob.cu"
    src.write_text(CODE)
    r = subprocess.run(["nvcc", *build.ARCH, "-std=c++17", "-DDDFAN_DD_FWD_CG=%d" % channels, "-I" + build.CSRC,
                        "-I" + build.ROOT + "/include", "-c", str(src), "-o", str(tmp_path / "knob.o")],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-800:]
