"""Builds with fewer wave lanes than the default (TR_WAVE_LANES): no render may take more lanes than there are."""
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "jarabotransientrendering_b200", "csrc")


@pytest.mark.parametrize("lanes", [1, 2, 3, 4])
def test_large_renders_take_the_lanes_there_are(tmp_path, lanes):
    src = tmp_path / "lanes.cu"
    src.write_text('#include "tr_internal.h"\n'
                   "static_assert(tri::large_lanes(true) >= 1 && tri::large_lanes(true) <= tri::kWaveLanes);\n"
                   "static_assert(tri::large_lanes(false) >= 1 && tri::large_lanes(false) <= tri::kWaveLanes);\n"
                   f"static_assert(tri::large_lanes(true) == {min(lanes, 3)} && tri::large_lanes(false) == {min(lanes, 2)});\n")
    r = subprocess.run(["nvcc", "-gencode", "arch=compute_100a,code=sm_100a", "-std=c++17", f"-DTR_WAVE_LANES={lanes}",
                        "-I", CSRC, "-I", os.path.join(CSRC, "..", "..", "include"), "-c", str(src), "-o",
                        str(tmp_path / "lanes.o")], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr
