"""CPU: the row cursors of the range PageRank's counting sort stay inside
their rows when the fill pass meets more or fewer edges than were counted."""
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent


@pytest.mark.parametrize("rows", [
    [(0, 0), (1, 1), (7, 7), (1000, 1000)],          # as counted
    [(0, 1), (0, 2), (0, 5), (1, 3), (4, 9)],        # edges added between the passes
    [(1, 0), (5, 2), (64, 63), (300, 1)],            # edges gone between the passes
])
def test_row_cursors_stay_in_their_rows(tmp_path, rows):
    exe = tmp_path / "rows"
    cxx = "/usr/bin/g++" if Path("/usr/bin/g++").exists() else "g++"
    r = subprocess.run([cxx, "-std=c++17", "-O1", "-Wall", "-Werror",
                        f"-I{ROOT / 'meerkat_b200' / 'csrc'}",
                        str(ROOT / "tests" / "cpp" / "row_cursor_driver.cpp"), "-o", str(exe)],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([str(exe)] + [str(x) for row in rows for x in row], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
