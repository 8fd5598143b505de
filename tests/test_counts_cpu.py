"""Host side of the exact polygon counts (no GPU): the modes written from a shell's orbits
are those of a walk over the whole grid, and enumeration is chosen by its cost."""
import os
import subprocess

from polyspectrum_b200 import build

HERE = os.path.dirname(os.path.abspath(__file__))


def test_lists_and_their_limits(tmp_path):
    exe = str(tmp_path / "count_lists")
    subprocess.run([build.nvcc(), *build.ARCH, "-O3", "-std=c++17", "-I", build.CSRC, "-o", exe,
                    os.path.join(HERE, "native", "count_lists.cu")], check=True)
    out = subprocess.run([exe], check=True, capture_output=True, text=True).stdout.splitlines()
    assert out[0] == "modes 0 of 322 wrong"
    rules = [line for line in out if line.startswith("rule")]
    assert len(rules) == 10
    for line in rules:
        got, want = line.split(": ", 1)[1].split(",")[0].split(" want ")
        assert got == want, line
