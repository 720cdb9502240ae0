"""rad_split.h, the places of a slab's corner-split lists: columns lie one after the
other without a gap, each with the room it can use."""
import pathlib
import shutil
import subprocess

import pytest

SRC = r"""
#include <cstdio>
#include <initializer_list>
#include "rad_split.h"
using namespace gfm;
int main() {
    long bad = 0;
    for (int DA = 1; DA <= 200; ++DA)
        for (int Dv : {2, 4, 62, 64, 66, 200, 400}) {
            int at = 0;
            for (int c = 1; c <= DA; ++c) {
                const int room = c == 1 || c == DA ? Dv : (Dv < 64 ? Dv : 64);
                bad += split_first(DA, Dv, c) != at || split_room(DA, Dv, c) != room;
                at += room;
            }
            bad += split_first(DA, Dv, DA + 1) != at;
        }
    std::printf("%ld\n", bad);
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_lists_lie_one_after_the_other(tmp_path):
    csrc = pathlib.Path(__file__).resolve().parent.parent / "gfm_gb300" / "csrc"
    (tmp_path / "s.cpp").write_text(SRC)
    subprocess.run(["g++", "-O2", "-std=c++17", f"-I{csrc}", "s.cpp", "-o", "s"], cwd=tmp_path, check=True)
    assert subprocess.run(["./s"], cwd=tmp_path, check=True, capture_output=True, text=True).stdout.strip() == "0"
