"""Builds ``pam_b200/libpam_b200.so`` — every CUDA source under ``pam_b200/csrc`` compiled for
sm_100a with nvcc and linked into one C-ABI shared library (declared in ``include/pam_b200.h``) —
and ``pam_b200/_host.so``, the host path of the operators (``csrc/host.cpp``, a CPython module over
torch's C++ headers that calls that library).

    python -m pam_b200.build [--force] [--verbose]

The kernel library does not depend on torch.  ``-fmad=false`` keeps nvcc from fusing a multiply into a
following add: the PAM kernels reproduce the reference's roundings operation by operation and
use explicit fused multiply-adds only where the reference's build does.
"""
import concurrent.futures
import pathlib
import shutil
import subprocess
import sys

PKG = pathlib.Path(__file__).resolve().parent
CSRC = PKG / "csrc"
OBJ = PKG / "build"
LIB = PKG / "libpam_b200.so"
HOST = PKG / "_host.so"
HOST_STAMP = OBJ / "host_platform.txt"

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
    "-fmad=false", "-Xcompiler", "-fPIC", "-Xcompiler", "-O2",
]


def _nvcc():
    exe = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not pathlib.Path(exe).exists():
        raise RuntimeError("nvcc not found: pam_b200 needs the CUDA toolkit to build its kernels")
    return exe


def _stale(target, deps):
    return not target.exists() or any(d.stat().st_mtime > target.stat().st_mtime for d in deps)


def _host_platform():
    """What the host module's binary depends on beside its sources: torch's C++ ABI and Python's."""
    import torch
    return f"torch {torch.__version__}, Python {sys.version_info.major}.{sys.version_info.minor}"


def host_stale():
    return (_stale(HOST, [CSRC / "host.cpp", PKG.parent / "include" / "pam_b200.h", pathlib.Path(__file__)])
            or not HOST_STAMP.exists() or HOST_STAMP.read_text() != _host_platform())


def build_host(force=False, verbose=False):
    """The CPython module with the operators' host path: plain C++, no device code."""
    import sysconfig

    import torch
    src = CSRC / "host.cpp"
    if not force and not host_stale():
        return HOST
    root = pathlib.Path(torch.__file__).resolve().parent
    cuda = pathlib.Path(_nvcc()).resolve().parents[1] / "include"
    cmd = ["g++", "-O2", "-std=c++17", "-fPIC", "-shared", f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
           *(f"-isystem{d}" for d in (root / "include", root / "include/torch/csrc/api/include", cuda, sysconfig.get_paths()["include"])),
           str(src), "-o", str(HOST), f"-L{root / 'lib'}", "-ltorch_python", "-ltorch", "-ltorch_cpu", "-ltorch_cuda",
           "-lc10", "-lc10_cuda", "-ldl"]
    res = subprocess.run(cmd, capture_output=True, text=True)
    if verbose or res.returncode:
        sys.stderr.write(res.stdout + res.stderr)
    if res.returncode:
        raise RuntimeError("g++ failed: " + " ".join(cmd))
    OBJ.mkdir(exist_ok=True)
    HOST_STAMP.write_text(_host_platform())
    return HOST


def build(force=False, verbose=False):
    sources = sorted(CSRC.glob("*.cu"))
    headers = sorted(CSRC.glob("*.cuh")) + [PKG.parent / "include" / "pam_b200.h", pathlib.Path(__file__)]
    OBJ.mkdir(exist_ok=True)
    nvcc = _nvcc()
    jobs = []
    for src in sources:
        obj = OBJ / (src.stem + ".o")
        if force or _stale(obj, [src, *headers]):
            cmd = [nvcc, *NVCC_FLAGS, "-c", str(src), "-o", str(obj)]
            if verbose:
                cmd.insert(1, "-Xptxas=-v")
            jobs.append(cmd)
    if jobs:
        with concurrent.futures.ThreadPoolExecutor(max_workers=8) as pool:
            for cmd, res in zip(jobs, pool.map(lambda c: subprocess.run(c, capture_output=True, text=True), jobs)):
                if verbose or res.returncode:
                    sys.stderr.write(res.stdout + res.stderr)
                if res.returncode:
                    raise RuntimeError("nvcc failed: " + " ".join(cmd))
    objs = [OBJ / (s.stem + ".o") for s in sources]
    if force or jobs or _stale(LIB, objs):
        subprocess.check_call([nvcc, "-shared", "-o", str(LIB), *map(str, objs), "-gencode",
                               "arch=compute_100a,code=sm_100a"])
    build_host(force, verbose)
    return LIB


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="--verbose" in sys.argv))
