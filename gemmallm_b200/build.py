"""Build libmoe_b200.so in-tree with nvcc for sm_100a, and the host extension
_host.so (csrc/host/, C++ against the installed torch and libmoe_b200.so).

    python -m gemmallm_b200.build [--force] [--verbose]

nvcc cross-compiles without a GPU. Objects go to gemmallm_b200/csrc/_build/,
the libraries to gemmallm_b200/ (git-ignored, built artefacts).
"""
from __future__ import annotations

import os
import importlib.util
import shutil
import subprocess
import sys
import sysconfig
from concurrent.futures import ThreadPoolExecutor
from pathlib import Path

PKG = Path(__file__).resolve().parent
CSRC = PKG / "csrc"
OBJ = CSRC / "_build"
LIB = PKG / "libmoe_b200.so"
HOST_SRC = CSRC / "host" / "host.cpp"
HOST_LIB = PKG / "_host.so"

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a",
    "-O3", "-std=c++17", "-lineinfo",
    "-Xcompiler", "-fPIC",
    "--expt-relaxed-constexpr",
]


def _nvcc() -> str:
    for cand in (os.environ.get("NVCC"), shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if cand and Path(cand).exists():
            return cand
    raise RuntimeError("nvcc not found: libmoe_b200.so cannot be built")


def sources() -> list[Path]:
    return sorted(CSRC.glob("*.cu"))


def _stale(target: Path, deps: list[Path]) -> bool:
    if not target.exists():
        return True
    t = target.stat().st_mtime
    return any(d.stat().st_mtime > t for d in deps)


def build(force: bool = False, verbose: bool = False) -> Path:
    nvcc = _nvcc()
    OBJ.mkdir(exist_ok=True)
    headers = sorted(CSRC.glob("*.cuh")) + [CSRC / "internal.h", PKG.parent / "include" / "moe_b200.h"]
    jobs = []
    objs = []
    for src in sources():
        obj = OBJ / (src.stem + ".o")
        objs.append(obj)
        if force or _stale(obj, [src] + headers):
            cmd = [nvcc, *NVCC_FLAGS, "-c", str(src), "-o", str(obj)]
            if verbose:
                cmd.insert(1, "-Xptxas")
                cmd.insert(2, "-v")
            jobs.append(cmd)

    def run(cmd):
        r = subprocess.run(cmd, capture_output=True, text=True)
        return cmd, r

    with ThreadPoolExecutor(max_workers=min(8, max(1, len(jobs)))) as ex:
        for cmd, r in ex.map(run, jobs):
            if verbose or r.returncode != 0:
                sys.stderr.write(" ".join(cmd) + "\n" + r.stdout + r.stderr)
            if r.returncode != 0:
                raise RuntimeError(f"nvcc failed on {cmd[-3]}")
    if force or jobs or _stale(LIB, objs):
        cmd = [nvcc, "-shared", "-o", str(LIB), *map(str, objs), "-cudart", "static"]
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode != 0:
            sys.stderr.write(r.stdout + r.stderr)
            raise RuntimeError("link of libmoe_b200.so failed")
    build_host(force, verbose)
    return LIB


def build_host(force: bool = False, verbose: bool = False) -> Path:
    """The modules' native host path: one C++ file against torch's headers, linked to
    libmoe_b200.so next to it."""
    deps = [HOST_SRC, CSRC / "internal.h", PKG.parent / "include" / "moe_b200.h"]
    torch_dir = Path(next(iter(importlib.util.find_spec("torch").submodule_search_locations)))
    # a library built against another torch's headers must not be loaded next to this one, whatever the files' dates
    stamp, version = OBJ / "host_torch_version", (torch_dir / "version.py").read_text()
    if not force and not _stale(HOST_LIB, deps) and stamp.exists() and stamp.read_text() == version:
        return HOST_LIB
    cuda = Path(_nvcc()).resolve().parent.parent
    includes = [torch_dir / "include", torch_dir / "include" / "torch" / "csrc" / "api" / "include",
                sysconfig.get_paths()["include"], cuda / "include"]
    cmd = [os.environ.get("CXX", "g++"), "-O2", "-std=c++17", "-fPIC", "-shared", *(f"-I{i}" for i in includes),
           str(HOST_SRC), "-o", str(HOST_LIB), f"-L{torch_dir / 'lib'}", "-ltorch", "-ltorch_cpu", "-ltorch_cuda",
           "-ltorch_python", "-lc10", "-lc10_cuda", f"-L{PKG}", f"-l:{LIB.name}", "-Wl,-rpath,$ORIGIN"]
    r = subprocess.run(cmd, capture_output=True, text=True)
    if verbose or r.returncode != 0:
        sys.stderr.write(" ".join(cmd) + "\n" + r.stdout + r.stderr)
    if r.returncode != 0:
        raise RuntimeError("build of _host.so failed")
    OBJ.mkdir(exist_ok=True)
    stamp.write_text(version)
    return HOST_LIB


if __name__ == "__main__":
    path = build(force="--force" in sys.argv, verbose="--verbose" in sys.argv)
    print(path)
