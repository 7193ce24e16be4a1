"""Build recipe for libanna_b200_kv.so (hand-written CUDA for sm_100a, no torch headers involved) and for the Python call
module on top of it.

``python -m anna_b200.build`` compiles every ``csrc/*.cu`` with nvcc (cross-compiles without a GPU) and links
them into ``anna_b200/libanna_b200_kv.so`` next to this file, so the library travels with the source tree; then
``csrc/launch_module.cpp`` with the host compiler against the installed torch into ``anna_b200/_launch.so``.
"""
from __future__ import annotations

import os
import shutil
import subprocess
import sys
from concurrent.futures import ThreadPoolExecutor
from pathlib import Path

PKG_DIR = Path(__file__).resolve().parent
CSRC = PKG_DIR / "csrc"
BUILD_DIR = PKG_DIR / "_build"
LIB_PATH = PKG_DIR / "libanna_b200_kv.so"
MODULE_SOURCE = CSRC / "launch_module.cpp"
MODULE_PATH = PKG_DIR / "_launch.so"
MODULE_STAMP = BUILD_DIR / "launch_module.stamp"  # what MODULE_PATH was built for

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a",
    "-lineinfo", "-O3", "-std=c++17",
    "-Xcompiler", "-fPIC",
    "-Xptxas=-v",
]


def _nvcc() -> str:
    found = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(found):
        raise RuntimeError("nvcc not found: libanna_b200_kv.so cannot be built")
    return found


def _stale(target: Path, sources: list[Path]) -> bool:
    if not target.exists():
        return True
    stamp = target.stat().st_mtime
    return any(src.stat().st_mtime > stamp for src in sources)


def module_stamp() -> str:
    """What the call module is compiled against besides its sources: it reads tensors and Python objects by the layout of the
    installed headers.  Compiled into the module as ``built_for``."""
    import torch

    return f"torch {torch.__version__}, cxx11 abi {int(torch._C._GLIBCXX_USE_CXX11_ABI)}, {sys.implementation.cache_tag}"


def build_module(force: bool = False, verbose: bool = False) -> Path:
    """The call module; needs the library, whose C entry points it links."""
    header = PKG_DIR.parent / "include" / "anna_b200_kv.h"
    stamp = module_stamp()
    current = MODULE_STAMP.exists() and MODULE_STAMP.read_text() == stamp
    if not force and current and not _stale(MODULE_PATH, [MODULE_SOURCE, header]):
        return MODULE_PATH
    import sysconfig

    import torch

    torch_dir = Path(torch.__file__).resolve().parent
    cuda_include = Path(_nvcc()).resolve().parent.parent / "include"
    includes = [header.parent, torch_dir / "include", torch_dir / "include" / "torch" / "csrc" / "api" / "include", cuda_include,
                sysconfig.get_paths()["include"]]
    cmd = [os.environ.get("CXX", "g++"), "-O2", "-std=c++17", "-fPIC", "-shared",
           f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}", f'-DANNA_BUILT_FOR="{stamp}"', *[f"-I{path}" for path in includes],
           str(MODULE_SOURCE), "-o", str(MODULE_PATH), f"-L{torch_dir / 'lib'}", "-ltorch_python", "-ltorch_cpu", "-lc10",
           "-lc10_cuda", f"-L{PKG_DIR}", f"-l:{LIB_PATH.name}", "-Wl,-rpath,$ORIGIN"]
    done = subprocess.run(cmd, capture_output=True, text=True)
    if done.returncode != 0:
        raise RuntimeError(f"{MODULE_SOURCE.name} failed:\n{done.stderr}")
    if verbose:
        sys.stderr.write(done.stderr)
    BUILD_DIR.mkdir(exist_ok=True)
    MODULE_STAMP.write_text(stamp)
    return MODULE_PATH


def build(force: bool = False, verbose: bool = False) -> Path:
    sources = sorted(CSRC.glob("*.cu"))
    headers = sorted(CSRC.glob("*.cuh")) + [PKG_DIR.parent / "include" / "anna_b200_kv.h"]
    BUILD_DIR.mkdir(exist_ok=True)
    nvcc = _nvcc()
    jobs = []
    for src in sources:
        obj = BUILD_DIR / (src.stem + ".o")
        if force or _stale(obj, [src, *headers]):
            jobs.append((src, obj))

    def compile_one(job: tuple[Path, Path]) -> str:
        src, obj = job
        cmd = [nvcc, *NVCC_FLAGS, "-c", str(src), "-o", str(obj)]
        done = subprocess.run(cmd, capture_output=True, text=True)
        if done.returncode != 0:
            raise RuntimeError(f"nvcc failed for {src.name}:\n{done.stderr}")
        return done.stderr

    with ThreadPoolExecutor(max_workers=min(8, max(1, len(jobs)))) as pool:
        logs = list(pool.map(compile_one, jobs))
    if verbose:
        for log in logs:
            sys.stderr.write(log)
    objects = [BUILD_DIR / (src.stem + ".o") for src in sources]
    if force or jobs or _stale(LIB_PATH, objects):
        cmd = [nvcc, "-shared", "-o", str(LIB_PATH), *map(str, objects), "-cudart", "shared"]
        done = subprocess.run(cmd, capture_output=True, text=True)
        if done.returncode != 0:
            raise RuntimeError(f"link failed:\n{done.stderr}")
    build_module(force, verbose)
    return LIB_PATH


if __name__ == "__main__":
    path = build(force="--force" in sys.argv, verbose="-v" in sys.argv)
    print(path)
