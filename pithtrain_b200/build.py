"""Build the native sm_100a library in-tree with nvcc (no JIT cache).

Every ``csrc/*.cu`` file is compiled to an object with
``-gencode arch=compute_100a,code=sm_100a -lineinfo`` and linked into
``pithtrain_b200/_lib/libpithb200.so``, which :mod:`pithtrain_b200._native` loads with ctypes. ``csrc/host_ops.cpp`` (the host side
of the operators that run in every layer, with torch's headers) becomes ``_lib/pith_host_ops.so``.
Objects are rebuilt only when their source (or a header) is newer; the host library also when its compiler command or torch, to
whose C++ ABI it is bound, is another one (``_lib/pith_host_ops.txt`` says of which it is).
"""

from __future__ import annotations

import os
import shutil
import subprocess
import sys
from concurrent.futures import ThreadPoolExecutor
from pathlib import Path

ROOT = Path(__file__).resolve().parent
CSRC = ROOT / "csrc"
LIBDIR = ROOT / "_lib"
LIBNAME = "libpithb200.so"

NVCC_FLAGS = [
    "-gencode",
    "arch=compute_100a,code=sm_100a",
    "-lineinfo",
    "-O3",
    "-std=c++17",
    "--use_fast_math",
    "-Xcompiler",
    "-fPIC",
    "-Xcompiler",
    "-fvisibility=hidden",
    "--expt-relaxed-constexpr",
]


def _nvcc() -> str:
    cand = os.environ.get("NVCC") or "/usr/local/cuda/bin/nvcc"
    return cand if os.path.exists(cand) else "nvcc"


def _cuda_include() -> Path:
    """Headers of the toolkit that nvcc belongs to."""
    return Path(shutil.which(_nvcc()) or "/usr/local/cuda/bin/nvcc").resolve().parent.parent / "include"


def _newest_header_mtime() -> float:
    return max((p.stat().st_mtime for p in list(CSRC.glob("*.cuh")) + list(CSRC.glob("*.h"))), default=0.0)


def lib_path() -> Path:
    return LIBDIR / LIBNAME


def host_ops_command(out: Path) -> list:
    """Compiler command of ``csrc/host_ops.cpp`` (torch's headers; no CUDA code)."""
    import sysconfig

    from torch.utils import cpp_extension

    # nvcc's host compiler, not $CXX: one that links its own libstdc++ in cannot share exceptions and streams with torch's
    return ["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-fvisibility=hidden", "-DTORCH_EXTENSION_NAME=pith_host_ops",
            *(f"-I{p}" for p in cpp_extension.include_paths()), f"-I{_cuda_include()}", f"-I{sysconfig.get_paths()['include']}",
            str(CSRC / "host_ops.cpp"), "-o", str(out), f"-L{cpp_extension.library_paths()[0]}",
            "-lc10", "-lc10_cuda", "-ltorch", "-ltorch_cpu", "-ltorch_python"]


def _host_ops_stamp(cmd: list) -> str:
    import torch

    return f"torch {torch.__version__}\n{' '.join(cmd)}\n"


def host_ops_stale(out: Path, src: Path, cmd: list) -> bool:
    stamp = out.with_suffix(".txt")
    return (not out.exists() or out.stat().st_mtime < src.stat().st_mtime
            or not stamp.exists() or stamp.read_text() != _host_ops_stamp(cmd))


def build(verbose: bool = False, force: bool = False, ptxas_info: bool = False, bounds_check: bool = False) -> Path:
    """Compile and link the library; returns its path. ``bounds_check`` builds ``libpithb200_checked.so`` with
    ``-DPT_BOUNDS_CHECK`` (index validation in the kernels that address memory through device-computed indices)."""
    LIBDIR.mkdir(exist_ok=True)
    objdir = LIBDIR / ("obj_checked" if bounds_check else "obj")
    objdir.mkdir(exist_ok=True)
    sources = sorted(CSRC.glob("*.cu"))
    hdr_m = _newest_header_mtime()
    jobs = []
    for src in sources:
        obj = objdir / (src.stem + ".o")
        stale = force or not obj.exists() or obj.stat().st_mtime < max(src.stat().st_mtime, hdr_m)
        if stale:
            cmd = [_nvcc(), *NVCC_FLAGS, *(["-DPT_BOUNDS_CHECK"] if bounds_check else []), "-c", str(src), "-o", str(obj)]
            if ptxas_info:
                cmd[1:1] = ["-Xptxas", "-v"]
            jobs.append((src, cmd))

    host_out, host_src = LIBDIR / "pith_host_ops.so", CSRC / "host_ops.cpp"
    host_cmd = host_ops_command(host_out)
    if force or host_ops_stale(host_out, host_src, host_cmd):
        jobs.append((host_src, host_cmd))

    def run(job):
        src, cmd = job
        res = subprocess.run(cmd, capture_output=True, text=True)
        return src, res

    if jobs:
        with ThreadPoolExecutor(max_workers=min(8, len(jobs))) as ex:
            for src, res in ex.map(run, jobs):
                if verbose or ptxas_info or res.returncode != 0:
                    sys.stderr.write(f"[build] {src.name}\n{res.stdout}{res.stderr}\n")
                if res.returncode != 0:
                    raise RuntimeError(f"compiler failed for {src}")
                if src == host_src:
                    host_out.with_suffix(".txt").write_text(_host_ops_stamp(host_cmd))
    out = LIBDIR / "libpithb200_checked.so" if bounds_check else lib_path()
    objs = [str(objdir / (s.stem + ".o")) for s in sources]
    need_link = any(src.suffix == ".cu" for src, _ in jobs) or not out.exists()
    if need_link:
        cmd = [_nvcc(), "-shared", "-o", str(out), *objs, "-lcudart_static", "-lrt", "-lpthread", "-ldl"]
        res = subprocess.run(cmd, capture_output=True, text=True)
        if res.returncode != 0:
            sys.stderr.write(res.stdout + res.stderr)
            raise RuntimeError("link failed")
    return out


if __name__ == "__main__":
    p = build(verbose=True, force="--force" in sys.argv, ptxas_info="--ptxas" in sys.argv,
              bounds_check="--bounds-check" in sys.argv)
    print(p)
