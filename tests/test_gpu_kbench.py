"""The stand-alone timing harness runs every one of its launches."""
import subprocess

import pytest

from polyspectrum_b200 import build

pytestmark = pytest.mark.gpu


def test_harness_runs_to_its_end():
    out = subprocess.run([build.build_kbench(), "1"], capture_output=True, text=True, timeout=300)
    assert out.returncode == 0, out.stderr
    for what in ("pass_y@512", "pass_y field@512 R=32", "pass_y field@512 R=8", "pair_z@384", "pair_counts"):
        assert what in out.stdout, out.stdout
