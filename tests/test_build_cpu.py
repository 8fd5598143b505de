"""Which objects a build compiles again."""
import os
import subprocess

import pytest

from polyspectrum_b200 import build


@pytest.fixture
def tree(tmp_path, monkeypatch):
    """One source and one header in a build tree of their own."""
    monkeypatch.setattr(build, "CSRC", str(tmp_path))
    (tmp_path / "one.cuh").write_text("inline int one() { return 1; }\n")
    (tmp_path / "one.cu").write_text('#include "one.cuh"\nint f() { return one(); }\n')
    obj = str(tmp_path / "one.o")

    def compile():
        cmd = build._compile_cmd("one.cu", obj)
        subprocess.run(cmd, check=True)
        build._record(obj, cmd)

    def stale():
        return build._stale(obj, build._compile_cmd("one.cu", obj))

    return tmp_path, obj, compile, stale


def test_objects_follow_their_files_and_their_command(tree, monkeypatch):
    path, obj, compile, stale = tree
    assert stale()
    compile()
    assert not stale()
    t = os.path.getmtime(obj) + 10
    os.utime(path / "one.cuh", (t, t))
    assert stale()
    os.utime(path / "one.cuh", (t - 20, t - 20))
    assert not stale()
    monkeypatch.setattr(build, "FLAGS", [f for f in build.FLAGS if f != "-O3"] + ["-O2"])
    assert stale()
    compile()
    assert not stale()
    os.remove(obj + ".cmd")
    assert stale()


def test_library_built_with_other_flags_is_out_of_date(monkeypatch):
    build.build(quiet=True)
    assert build.up_to_date()
    monkeypatch.setattr(build, "FLAGS", [*build.FLAGS, "-DOTHER"])
    assert not build.up_to_date()
