"""Build ``libmoda_b200.so`` in-tree with nvcc for sm_100a.

    python -m moda_b200.build [--force] [--verbose]

The library is a plain C-ABI shared object (no torch, no pybind).  Beside it ``_native.so`` is built,
the PyTorch binding (``csrc/torch_binding.cpp``), which links against it and against torch.  Each is
rebuilt when the hash of the files it is built from (and of the compiler flags) differs from the one
in the stamp file beside the ``.so``.  Builds are serialised by a lock file and the library is
moved into place in one piece, so the ranks of a multi-GPU launch can all call ``build()``.

``build_wait_test()`` compiles the same sources with ``-DMODA_WAIT_TEST`` into
``libmoda_b200_waittest.so``: a test-only build in which the tcgen05 forwards and the dq /
dk/dv kernels withhold one barrier arrival and every bounded wait gives up after about a
millisecond, so that the wait-expiry teardown path can be exercised on a GPU without hanging it.  The
product never loads that file.
"""
from __future__ import annotations

import fcntl
import glob
import hashlib
import os
import shutil
import subprocess
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
CSRC = os.path.join(HERE, "csrc")
OUT = os.path.join(HERE, "libmoda_b200.so")
OUT_NATIVE = os.path.join(HERE, "_native.so")
BINDING = os.path.join(CSRC, "torch_binding.cpp")
OUT_WAIT_TEST = os.path.join(HERE, "libmoda_b200_waittest.so")

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a",
    "-lineinfo", "-O3", "-std=c++17",
    "-shared", "-Xcompiler", "-fPIC",
]


def sources():
    return sorted(glob.glob(os.path.join(CSRC, "*.cu")))


def _digest(extra, out: str = OUT) -> str:
    """Hash of everything a library is built from: sources, headers, compiler flags."""
    h = hashlib.sha256()
    h.update(" ".join(NVCC_FLAGS + list(extra)).encode())
    headers = glob.glob(os.path.join(ROOT, "include", "*.h"))
    if out == OUT_NATIVE:
        import torch
        h.update(torch.__version__.encode())
        deps = [BINDING] + headers
    else:
        deps = [f for f in glob.glob(os.path.join(CSRC, "*")) if f != BINDING] + headers
    for d in sorted(deps):
        if os.path.isfile(d):
            h.update(os.path.basename(d).encode())
            with open(d, "rb") as f:
                h.update(f.read())
    return h.hexdigest()


def _stale(out: str = OUT, extra=()) -> bool:
    """The library is current when the stamp beside it holds the hash of the present sources.
    File times play no part: a checkout or a copy of the tree changes them without changing a byte."""
    stamp = out + ".stamp"
    if not (os.path.exists(out) and os.path.exists(stamp)):
        return True
    with open(stamp) as f:
        return f.read().strip() != _digest(extra, out)


def _nvcc_command(tmp: str, extra, verbose: bool):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    return [nvcc] + NVCC_FLAGS + list(extra) + (["-Xptxas", "-v"] if verbose else []) + ["-o", tmp] + sources()


def _binding_command(tmp: str):
    import sysconfig

    import torch
    t = os.path.join(os.path.dirname(torch.__file__))
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    cuda = os.path.dirname(os.path.dirname(os.path.realpath(nvcc)))
    return ["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-fvisibility=hidden",
            f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
            "-isystem", os.path.join(t, "include"), "-isystem", os.path.join(t, "include", "torch", "csrc", "api", "include"),
            "-isystem", os.path.join(cuda, "include"), "-isystem", sysconfig.get_paths()["include"], BINDING, "-o", tmp,
            "-L" + HERE, "-l:libmoda_b200.so", "-L" + os.path.join(t, "lib"), "-lc10", "-lc10_cuda", "-ltorch", "-ltorch_cpu",
            "-ltorch_python", "-Wl,-rpath,$ORIGIN"]


def _compile(out: str, extra, force: bool, command) -> str:
    if not force and not _stale(out, extra):
        return out
    # One builder at a time, and the file appears in one piece: the ranks of a multi-GPU launch all
    # come here, and a library that another process is still writing must never be loaded.
    with open(out + ".lock", "w") as lock:
        fcntl.flock(lock, fcntl.LOCK_EX)
        try:
            if not force and not _stale(out, extra):      # built by another process in the meantime
                return out
            tmp = f"{out}.tmp.{os.getpid()}"
            res = subprocess.run(command(tmp), capture_output=True, text=True)
            if res.returncode != 0 or "-v" in command(tmp):
                sys.stderr.write(res.stdout + res.stderr)
            if res.returncode != 0:
                if os.path.exists(tmp):
                    os.remove(tmp)
                raise RuntimeError("building " + os.path.basename(out) + " failed")
            os.replace(tmp, out)
            with open(out + ".stamp.tmp", "w") as f:
                f.write(_digest(extra, out) + "\n")
            os.replace(out + ".stamp.tmp", out + ".stamp")
        finally:
            fcntl.flock(lock, fcntl.LOCK_UN)
    return out


def build(force: bool = False, verbose: bool = False) -> str:
    _compile(OUT, [], force, lambda tmp: _nvcc_command(tmp, [], verbose))
    _compile(OUT_NATIVE, [], force, _binding_command)       # links against the library
    return OUT


def build_wait_test(force: bool = False, verbose: bool = False) -> str:
    extra = ["-DMODA_WAIT_TEST"]
    return _compile(OUT_WAIT_TEST, extra, force, lambda tmp: _nvcc_command(tmp, extra, verbose))


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="--verbose" in sys.argv))
    if "--wait-test" in sys.argv:
        print(build_wait_test(force="--force" in sys.argv))
