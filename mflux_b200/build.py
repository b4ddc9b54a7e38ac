"""In-tree build of libmfx.so (sm_100a only) with nvcc and of the host module _host.so with g++. No GPU is needed to build.

Usage: python -m mflux_b200.build [--force] [--verbose]
Objects are rebuilt only when their source (or a header) is newer. The shared libraries land next
to this file so that they travel with the source tree.
"""
from __future__ import annotations

import importlib.util
import os
import shutil
import subprocess
import sys
import sysconfig
from concurrent.futures import ThreadPoolExecutor
from pathlib import Path

PKG = Path(__file__).resolve().parent
CSRC = PKG / "csrc"
OBJ = PKG / "build"
LIB = PKG / "libmfx.so"
HOST = PKG / "_host.so"
ROOT = PKG.parent

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a",
    "-O3", "-std=c++17", "-lineinfo",
    "-Xcompiler", "-fPIC",
    "--expt-relaxed-constexpr",
    "-Xptxas", "-v",
    "-DMFX_BUILDING",
]


def _nvcc() -> str:
    cand = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(cand):
        raise RuntimeError("nvcc not found; libmfx.so cannot be built")
    return cand


def sources() -> list[Path]:
    return sorted(CSRC.glob("*.cu"))


def _stale(obj: Path, src: Path, headers: list[Path]) -> bool:
    if not obj.exists():
        return True
    t = obj.stat().st_mtime
    return any(p.stat().st_mtime > t for p in [src, *headers])


def host_builds_for() -> str:
    """What the host module is tied to: the torch build whose inlined tensor layouts it has, and the Python ABI."""
    spec = importlib.util.spec_from_file_location("_torch_version", _torch() / "version.py")
    version = importlib.util.module_from_spec(spec)     # without importing torch itself
    spec.loader.exec_module(version)
    return f"torch {version.__version__} {sysconfig.get_config_var('SOABI')}"


def _torch() -> Path:
    return Path(importlib.util.find_spec("torch").origin).parent


def build_host(force: bool, headers: list[Path]) -> None:
    """The CPython module of csrc/host_call.cpp, against the headers and libraries of the installed torch. Stale, too, when
    it was built for another torch or Python; the module carries the same text for the loader to compare."""
    src, record = CSRC / "host_call.cpp", OBJ / "_host.built_for"
    built_for = host_builds_for()
    known = record.read_text() if record.exists() else None
    if not force and known == built_for and not _stale(HOST, src, headers):
        return
    torch = _torch()
    cuda = Path(_nvcc()).resolve().parent.parent
    record.unlink(missing_ok=True)     # nothing is known about what a failure below leaves
    cmd = [shutil.which("g++") or "c++", "-O2", "-std=c++17", "-fPIC", "-shared", "-Wall", f'-DMFX_BUILT_FOR="{built_for}"',
           "-I", str(ROOT / "include"), "-I", str(torch / "include"), "-I", str(torch / "include/torch/csrc/api/include"),
           "-I", str(cuda / "include"), "-I", sysconfig.get_paths()["include"], str(src), "-o", str(HOST),
           "-L", str(torch / "lib"), "-ltorch_python", "-ltorch_cpu", "-lc10", "-lc10_cuda"]
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError(f"build of {HOST.name} failed:\n{r.stdout}\n{r.stderr}")
    record.write_text(built_for)


def build(force: bool = False, verbose: bool = False) -> Path:
    nvcc = _nvcc()
    OBJ.mkdir(exist_ok=True)
    headers = sorted(CSRC.glob("*.cuh")) + sorted((ROOT / "include").glob("*.h"))
    jobs = []
    for src in sources():
        obj = OBJ / (src.stem + ".o")
        if force or _stale(obj, src, headers):
            jobs.append((src, obj))

    def compile_one(job):
        src, obj = job
        cmd = [nvcc, *NVCC_FLAGS, "-I", str(ROOT / "include"), "-c", str(src), "-o", str(obj)]
        r = subprocess.run(cmd, capture_output=True, text=True)
        (OBJ / (src.stem + ".ptxas.log")).write_text(r.stderr)
        if r.returncode != 0:
            raise RuntimeError(f"nvcc failed for {src.name}:\n{r.stdout}\n{r.stderr}")
        if verbose:
            print(r.stderr)
        return obj

    if jobs:
        with ThreadPoolExecutor(max_workers=min(8, len(jobs))) as ex:
            list(ex.map(compile_one, jobs))
    objs = [OBJ / (s.stem + ".o") for s in sources()]
    if jobs or not LIB.exists():
        cmd = [nvcc, "-shared", "-o", str(LIB), *map(str, objs), "-lcudart_static", "-lpthread", "-ldl", "-lrt"]
        cmd[1:1] = ["-gencode", "arch=compute_100a,code=sm_100a", "-Xcompiler", "-fPIC"]
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode != 0:
            raise RuntimeError(f"link failed:\n{r.stdout}\n{r.stderr}")
    build_host(force, headers)
    return LIB


if __name__ == "__main__":
    out = build(force="--force" in sys.argv, verbose="--verbose" in sys.argv)
    print(out)
