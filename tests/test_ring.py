"""feed_ring (csrc/hg_ring.h), the order of waits and copies of the weight
gradients' copying thread, compiled for the host with simulated barriers."""
import ctypes as C
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "bevy_hair_gb300" / "csrc"
STAGES = 6

SOURCE = """
#include <vector>
#include "hg_ring.h"

// Readers that take `read` tiles and then give up; copies whose stage is
// `stuck` never land.  Returns the copies neither landed nor waited for, with
// 1000 added when feed_ring reported success and 10000 for a wait of another
// phase than the stage's last copy's.
extern "C" int run(unsigned tiles, unsigned read, unsigned stuck) {
    constexpr unsigned kStages = %d;
    std::vector<int> under_way(kStages, -1);  // the tile being copied into a stage
    int wrong = 0;
    auto land = [&](unsigned s) { if (s != stuck) under_way[s] = -1; };
    const bool ok = hg::feed_ring<kStages>(
        tiles,
        [&](unsigned s, unsigned parity) {
            const int before = under_way[s];  // a stage is empty when its readers saw its tile
            if (before >= 0 && ((before / kStages) & 1u) != parity) wrong = 1;
            if (before < 0 || (unsigned)before >= read || s == stuck) return false;
            land(s);
            return true;
        },
        [&](unsigned s, unsigned tile) {
            if (under_way[s] >= 0) wrong = 1;
            under_way[s] = (int)tile;
        },
        [&](unsigned s, unsigned parity) {
            if (under_way[s] < 0 || ((under_way[s] / kStages) & 1u) != parity) wrong = 1;
            if (s == stuck) { under_way[s] = -1; return false; }  // the wait itself ran out
            land(s);
            return true;
        });
    int left = 0;
    for (int t : under_way) left += t >= 0;
    return left + (ok ? 1000 : 0) + (wrong ? 10000 : 0);
}
""" % STAGES


@pytest.fixture(scope="module")
def ring(tmp_path_factory):
    d = tmp_path_factory.mktemp("ring")
    (d / "ring.cpp").write_text(SOURCE)
    subprocess.run(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", f"-I{CSRC}", "-o", str(d / "ring.so"),
                    str(d / "ring.cpp")], check=True)
    return C.CDLL(str(d / "ring.so")).run


@pytest.mark.parametrize("tiles", [1, 5, 6, 7, 12, 16])
def test_every_copy_is_waited_for(ring, tiles):
    """The readers give up after any number of tiles, or a copy never lands:
    the thread reports it and leaves no copy behind it."""
    nobody = STAGES
    for read in range(tiles + 1):
        needed = max(tiles - STAGES, 0)  # tiles whose stage is filled again
        assert ring(tiles, read, nobody) == (1000 if read >= needed else 0), (tiles, read)
    for stuck in range(min(STAGES, tiles)):
        assert ring(tiles, tiles, stuck) == 0, (tiles, stuck)
