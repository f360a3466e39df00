"""The numbering of the grid-line sweeps' tiles (csrc/line_tiles.h) on the CPU."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_tiles_by_brute_force(tmp_path):
    exe = str(tmp_path / "line_tiles_test")
    subprocess.run(["g++", "-std=c++17", "-O2", "-Wall", "-Werror",
                    "-I" + os.path.join(ROOT, "mtl4-mirror_b200", "csrc"),
                    os.path.join(ROOT, "tests", "cpp", "line_tiles_test.cpp"), "-o", exe],
                   check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout
