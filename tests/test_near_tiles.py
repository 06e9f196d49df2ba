"""The tiled search of the near lists: every panel of a list is found in exactly
one tile, and every panel that is missing is reported by exactly one, also where
it lies between the last panel of a tile and the first of the next."""
import pathlib
import shutil
import subprocess

CSRC = pathlib.Path(__file__).resolve().parent.parent / "hornsculpt_b200" / "csrc"
SOURCE = r"""
#include "near_tiles.cuh"
#include <cstdio>
#include <random>
#include <vector>
int main() {
    std::mt19937 rng(3);
    long boundary = 0;
    for (int trial = 0; trial < 4000; ++trial) {
        const uint32_t panels = 1 + rng() % 60, tile = 1 + rng() % 9, keep = rng() % 101;
        std::vector<uint32_t> list;
        std::vector<bool> has(panels, false);
        for (uint32_t s = 0; s < panels; ++s)
            if (rng() % 100 < keep) {
                list.push_back(s);
                has[s] = true;
            }
        const uint32_t length = list.size();
        for (uint32_t s = 0; s < panels; ++s) {
            int found = 0, missed = 0;
            for (uint32_t base = 0; base == 0 || base < length; base += tile) {  // as the kernel's loop
                const uint32_t count = std::min(tile, length - base), previous = base ? list[base - 1] : 0;
                const uint32_t *t = list.data() + base;
                const uint32_t at = hsb::nearTilePlace(t, count, s);
                if (at < count && t[at] == s)
                    ++found;
                else
                    missed += hsb::nearTileMisses(at, count, base == 0, base + count >= length, previous, s);
                if (base && !has[s] && s > previous && s < t[0])
                    ++boundary;
            }
            if (found != (has[s] ? 1 : 0) || missed != (has[s] ? 0 : 1)) {
                std::printf("panel %u of %u, tile %u: found %d, missed %d\n", s, length, tile, found, missed);
                return 1;
            }
        }
    }
    return boundary > 1000 ? 0 : 2;
}
"""


def test_a_missing_panel_is_always_reported(tmp_path):
    (tmp_path / "tiles.cpp").write_text(SOURCE)
    subprocess.run([shutil.which("g++") or "c++", "-std=c++20", "-O2", "-include", "algorithm", "-I", str(CSRC),
                    str(tmp_path / "tiles.cpp"), "-o", str(tmp_path / "tiles")], check=True)
    run = subprocess.run([str(tmp_path / "tiles")], capture_output=True, text=True)
    assert run.returncode == 0, run.stdout
