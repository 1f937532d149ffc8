"""The launch count that bench.py reports for a frame."""
import re
import sys
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]
sys.path.insert(0, str(ROOT))

import bench  # noqa: E402


@pytest.mark.parametrize("strands, side, sms, launches", [
    (300, 32, 152, 10), (300, 0, 152, 7),               # one camera stage
    (7_296, 256, 152, 10), (7_297, 256, 152, 12), (7_297, 0, 152, 9),
    (32_767, 1024, 152, 12), (32_768, 1024, 152, 13),   # a front plane
    (40_000, 512, 152, 12), (40_000, 2048, 152, 12), (65_536, 2048, 152, 13), (100_000, 1024, 152, 13),
    (7_000, 256, 132, 12),
])
def test_frame_launches(strands, side, sms, launches):
    assert bench.frame_launches(strands, side, side, sms) == launches


def test_frame_launches_follow_the_library_s_rules():
    """The lines that frame_launches repeats, as the library has them."""
    csrc = ROOT / "bevy_hair_gb300" / "csrc"
    internal, raster = (csrc / "hg_internal.h").read_text(), (csrc / "raster.cu").read_text()

    def constant(text, name):
        return eval(re.search(rf"\b{name} = ([0-9 *+]+)[,;]", text).group(1))

    assert constant(internal, "kPlaneMinStrands") == 32768
    assert constant(internal, "kPlaneMinTexels") == 512 * 512 + 1
    assert constant(internal, "kPlaneTexelsPerStrand") == 64
    warps = constant(raster, "kRasterWarps") * int(re.search(r"return MODE == 0 \? (\d+)", raster).group(1))
    assert constant(raster, "kOneStageRounds") * warps == 48
