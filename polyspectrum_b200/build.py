"""Build libpsgpu.so (sm_100a) in-tree.

    python -m polyspectrum_b200.build [--force] [--ptxas-verbose] [--kbench]

Each translation unit compiles in its own nvcc process (the FFT kernels are
heavily unrolled); objects go to polyspectrum_b200/_build/, the shared library
to polyspectrum_b200/libpsgpu.so.  The library links the CUDA runtime
statically and depends on no torch symbol.  The command-line driver
(driver/ps_run.c, plain C over the C-ABI) is linked against it as
polyspectrum_b200/ps_run, and the ini-file generator (driver/ps_create_ini.c) as
polyspectrum_b200/ps_create_ini.  --kbench also builds polyspectrum_b200/ps_kbench, a
stand-alone timing harness of the hot passes (csrc/ps_kbench.cu).
"""
from __future__ import annotations

import argparse
import glob
import os
import shutil
import subprocess
import sys

PKG = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(PKG)
CSRC = os.path.join(PKG, "csrc")
OUT_DIR = os.path.join(PKG, "_build")
LIB = os.path.join(PKG, "libpsgpu.so")
DRIVER_SRC = os.path.join(PKG, "driver", "ps_run.c")
DRIVER = os.path.join(PKG, "ps_run")
KBENCH = os.path.join(PKG, "ps_kbench")
CREATE_INI_SRC = os.path.join(PKG, "driver", "ps_create_ini.c")
CREATE_INI = os.path.join(PKG, "ps_create_ini")
SOURCES = ["ps_inst_f32_a.cu", "ps_inst_f32_b.cu", "ps_inst_f32_mixed.cu", "ps_inst_f64_mixed.cu", "ps_inst_f64_a.cu",
           "ps_api.cu", "ps_inst_f32_c.cu", "ps_inst_f64_b.cu", "ps_inst_f64_c.cu", "ps_noalloc.cu"]

ARCH = ["-gencode", "arch=compute_100a,code=sm_100a"]
FLAGS = ARCH + ["-O3", "-lineinfo", "-std=c++17", "-Xcompiler", "-fPIC,-ffp-contract=off"]


def nvcc() -> str:
    for cand in (os.environ.get("NVCC"), shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if cand and os.path.exists(cand):
            return cand
    raise RuntimeError("nvcc not found")


def _deps() -> list[str]:
    return (glob.glob(os.path.join(CSRC, "*.cu")) + glob.glob(os.path.join(CSRC, "*.cuh"))
            + glob.glob(os.path.join(ROOT, "include", "*.h")))


def _compile_cmd(src: str, obj: str) -> list[str]:
    return [nvcc(), *FLAGS, "-MD", "-MF", obj + ".d", "-c", os.path.join(CSRC, src), "-o", obj]


def _signature(cmd: list[str]) -> str:
    """What an object's or the library's code depends on besides its files: the compiler and its options."""
    version = subprocess.run([cmd[0], "--version"], capture_output=True, text=True).stdout
    return "\n".join([*(a.replace(ROOT, ".") for a in cmd), version])  # (the same wherever the tree lies)


def _recorded(path: str, cmd: list[str]) -> bool:
    """Whether `path` was made by this command (kept beside it when it was made)."""
    if not os.path.exists(path + ".cmd"):
        return False
    with open(path + ".cmd") as f:
        return f.read() == _signature(cmd)


def _record(path: str, cmd: list[str]) -> None:
    with open(path + ".cmd", "w") as f:
        f.write(_signature(cmd))


def _stale(obj: str, cmd: list[str]) -> bool:
    """Whether an object is older than a file it was compiled from (nvcc's own
    dependency list), or was compiled by another command."""
    dep = obj + ".d"
    if not os.path.exists(obj) or not os.path.exists(dep) or not _recorded(obj, cmd):
        return True
    with open(dep) as f:
        files = f.read().split(":", 1)[1].replace("\\\n", " ").split()
    t = os.path.getmtime(obj)
    return any(not os.path.exists(p) or os.path.getmtime(p) > t for p in files)


def up_to_date() -> bool:
    if not os.path.exists(LIB):
        return False
    t = os.path.getmtime(LIB)
    if any(os.path.getmtime(p) > t for p in _deps()):
        return False
    objs = [os.path.join(OUT_DIR, src.replace(".cu", ".o")) for src in SOURCES]
    return all(_recorded(obj, _compile_cmd(src, obj)) for src, obj in zip(SOURCES, objs))


def build_driver(force: bool = False) -> str:
    """gcc the C driver against libpsgpu.so (rpath $ORIGIN: the two stay side by side)."""
    if (not force and os.path.exists(DRIVER)
            and os.path.getmtime(DRIVER) >= max(os.path.getmtime(DRIVER_SRC), os.path.getmtime(LIB),
                                                os.path.getmtime(os.path.join(ROOT, "include", "ps_gpu.h")))):
        return DRIVER
    tmp = DRIVER + ".tmp"
    subprocess.run(["gcc", "-std=c99", "-O2", "-Wall", "-Wextra", "-o", tmp, DRIVER_SRC, "-L", PKG, "-lpsgpu",
                    "-Wl,-rpath,$ORIGIN", "-lm"], check=True)
    os.replace(tmp, DRIVER)
    build_create_ini()
    return DRIVER


def build_create_ini() -> str:
    """gcc the ini-file generator (plain C, no library)."""
    if os.path.exists(CREATE_INI) and os.path.getmtime(CREATE_INI) >= os.path.getmtime(CREATE_INI_SRC):
        return CREATE_INI
    tmp = CREATE_INI + ".tmp"
    subprocess.run(["gcc", "-std=c99", "-O2", "-Wall", "-Wextra", "-o", tmp, CREATE_INI_SRC], check=True)
    os.replace(tmp, CREATE_INI)
    return CREATE_INI


def build(force: bool = False, ptxas_verbose: bool = False, quiet: bool = False) -> str:
    if not force and up_to_date():
        build_driver()
        return LIB
    os.makedirs(OUT_DIR, exist_ok=True)
    exe = nvcc()
    procs = []
    objs = []
    for src in SOURCES:
        obj = os.path.join(OUT_DIR, src.replace(".cu", ".o"))
        objs.append(obj)
        cmd = _compile_cmd(src, obj)
        if not force and not ptxas_verbose and not _stale(obj, cmd):
            continue
        extra = ["-Xptxas", "-v"] if ptxas_verbose else []
        if os.path.exists(obj + ".cmd"):
            os.remove(obj + ".cmd")
        procs.append((src, obj, cmd, subprocess.Popen(cmd + extra, stdout=subprocess.PIPE, stderr=subprocess.STDOUT,
                                                      text=True)))
    failed = False
    for src, obj, cmd, p in procs:
        out, _ = p.communicate()
        if p.returncode != 0:
            failed = True
            sys.stderr.write(f"nvcc failed for {src}:\n{out}\n")
            continue
        _record(obj, cmd)
        if out and (ptxas_verbose or not quiet):
            lines = [ln for ln in out.splitlines() if "Wno-deprecated" not in ln]
            if lines:
                sys.stdout.write("\n".join(lines) + "\n")
    if failed:
        raise RuntimeError("libpsgpu build failed")
    tmp = LIB + ".tmp"
    subprocess.run([exe, *ARCH, "-shared", "-cudart", "static", *objs, "-o", tmp], check=True)
    os.replace(tmp, LIB)
    build_driver(force=True)
    return LIB


def build_kbench() -> str:
    """nvcc the stand-alone kernel timing harness (no library link)."""
    tmp = KBENCH + ".tmp"
    subprocess.run([nvcc(), *FLAGS, "-o", tmp, os.path.join(CSRC, "ps_kbench.cu")], check=True)
    os.replace(tmp, KBENCH)
    return KBENCH


def main() -> None:
    ap = argparse.ArgumentParser()
    ap.add_argument("--force", action="store_true")
    ap.add_argument("--ptxas-verbose", action="store_true")
    ap.add_argument("--kbench", action="store_true")
    a = ap.parse_args()
    print(build(force=a.force, ptxas_verbose=a.ptxas_verbose))
    if a.kbench:
        print(build_kbench())


if __name__ == "__main__":
    main()
