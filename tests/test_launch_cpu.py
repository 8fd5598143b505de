"""Host-side checks of the launch wrappers (no GPU: every call is refused before it
reaches the device)."""
import os
import subprocess

from polyspectrum_b200 import build

HERE = os.path.dirname(os.path.abspath(__file__))


def test_launch_without_its_table_is_refused(tmp_path):
    build.build(quiet=True)
    exe = str(tmp_path / "launch_tables")
    subprocess.run([build.nvcc(), *build.ARCH, "-std=c++17", "-I", build.CSRC, "-o", exe,
                    os.path.join(HERE, "native", "launch_tables.cu"), "-L", build.PKG, "-lpsgpu",
                    "-Xlinker", f"-rpath={build.PKG}"], check=True)
    out = subprocess.run([exe], check=True, capture_output=True, text=True).stdout.splitlines()
    assert len(out) == 4 * 12
    for line in out:
        what, status, message = line.split("|", 2)
        assert int(status) < 0, line
        assert "twiddle table" in message, line
