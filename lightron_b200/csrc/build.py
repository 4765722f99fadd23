"""Builds the in-tree CUDA library with nvcc for sm_100a only.

    python -m lightron_b200.csrc.build [--verbose] [--force] [--sanitize]

The result, ``liblightron_b200.so``, sits beside the sources (git-ignored) and is loaded through
ctypes by ``lightron_b200.ops.native``.  No torch headers are involved in it, so it takes
seconds and cross-compiles on a machine without a GPU.  ``_host_ops.so`` (``host_ops.cpp``, the autograd nodes
that call it) is built against the installed torch, at the same time.

``--sanitize`` builds ``liblightron_b200_asan.so`` instead: the same sources with the HOST code under
AddressSanitizer + UndefinedBehaviorSanitizer (device code is unchanged).  Load it with
``LD_PRELOAD=$(gcc -print-file-name=libasan.so)``, ``ASAN_OPTIONS=detect_leaks=0:protect_shadow_gap=0`` and
``LIGHTRON_B200_LIB=<that file>``; ``tests/test_grouped_cpu.py`` runs the host-only entry points that way.
"""
from __future__ import annotations

import glob
import os
import subprocess
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
LIB = os.path.join(HERE, "liblightron_b200.so")
HOST_SRC, HOST_LIB = os.path.join(HERE, "host_ops.cpp"), os.path.join(HERE, "_host_ops.so")
ARCH = ["-gencode", "arch=compute_100a,code=sm_100a"]


def sources():
    return sorted(glob.glob(os.path.join(HERE, "*.cu")))


def host_tag() -> str:
    """What ``_host_ops.so`` is built against, as it is written into the file: classes of another torch have another layout."""
    import torch
    return f"lightron_b200 host ops: torch {torch.__version__}, python {sys.version_info[0]}.{sys.version_info[1]}."


def host_built_for_this_torch() -> bool:
    if not os.path.exists(HOST_LIB):
        return False
    with open(HOST_LIB, "rb") as f:
        return host_tag().encode() in f.read()


def host_command(out: str) -> list:
    """Compiler call for the extension module of the autograd nodes."""
    import sysconfig
    import torch
    base = os.path.dirname(torch.__file__)
    inc = [os.path.join(base, "include"), os.path.join(base, "include", "torch", "csrc", "api", "include"), sysconfig.get_paths()["include"],
           os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")]
    return [os.environ.get("CXX", "g++"), "-O2", "-std=c++17", "-fPIC", "-shared", "-fvisibility=hidden",
            f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}", f'-DLB_BUILT_FOR="{host_tag()}"', *(f"-I{d}" for d in inc), HOST_SRC, "-o", out,
            f"-L{os.path.join(base, 'lib')}", "-lc10", "-lc10_cuda", "-ltorch", "-ltorch_cpu", "-ltorch_python"]


def needs_build() -> bool:
    if not os.path.exists(LIB) or not host_built_for_this_torch():
        return True
    t = min(os.path.getmtime(LIB), os.path.getmtime(HOST_LIB))
    deps = sources() + [HOST_SRC] + glob.glob(os.path.join(HERE, "*.cuh")) + glob.glob(os.path.join(HERE, "*.h"))
    return any(os.path.getmtime(s) > t for s in deps)


def build(verbose: bool = False, force: bool = False) -> str:
    if not force and not needs_build():
        return LIB
    nvcc = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")
    objs, procs = [], []
    for src in sources():                      # one nvcc per source, all at once
        obj = src[:-3] + ".o"
        cmd = [nvcc, *ARCH, "-O3", "-lineinfo", "-std=c++17", "--use_fast_math", "-Xcompiler", "-fPIC", "-c", src, "-o", obj]
        if verbose:
            cmd.insert(1, "-Xptxas")
            cmd.insert(2, "-v")
        procs.append((src, subprocess.Popen(cmd, stdout=subprocess.PIPE, stderr=subprocess.PIPE, text=True)))
        objs.append(obj)
    procs.append((HOST_SRC, subprocess.Popen(host_command(HOST_LIB + ".tmp"), stdout=subprocess.PIPE, stderr=subprocess.PIPE, text=True)))
    failed = []
    for src, pr in procs:
        out, err = pr.communicate()
        if verbose or pr.returncode:
            sys.stderr.write(out + err)
        if pr.returncode:
            failed.append(os.path.basename(src))
    if failed:
        raise RuntimeError(f"compilation failed on {', '.join(failed)}")
    cmd = [nvcc, *ARCH, "-shared", "-o", LIB + ".tmp", *objs, "-lcudart"]
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode:
        sys.stderr.write(r.stdout + r.stderr)
        raise RuntimeError("link failed")
    os.replace(LIB + ".tmp", LIB)
    os.replace(HOST_LIB + ".tmp", HOST_LIB)
    return LIB


ASAN_LIB = os.path.join(HERE, "liblightron_b200_asan.so")
_SAN = ["-Xcompiler", "-fsanitize=address", "-Xcompiler", "-fsanitize=undefined", "-Xcompiler", "-fno-omit-frame-pointer"]


def build_sanitized(out: str = ASAN_LIB) -> str:
    """Host code under ASan + UBSan (objects go to a temporary directory; the normal build is untouched)."""
    import tempfile
    nvcc = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")
    with tempfile.TemporaryDirectory() as tmp:
        procs, objs = [], []
        for src in sources():
            obj = os.path.join(tmp, os.path.basename(src)[:-3] + ".o")
            cmd = [nvcc, *ARCH, "-O1", "-g", "-std=c++17", "--use_fast_math", "-Xcompiler", "-fPIC", *_SAN, "-c", src, "-o", obj]
            procs.append((src, subprocess.Popen(cmd, stdout=subprocess.PIPE, stderr=subprocess.PIPE, text=True)))
            objs.append(obj)
        for src, pr in procs:
            so, se = pr.communicate()
            if pr.returncode:
                sys.stderr.write(so + se)
                raise RuntimeError(f"nvcc (sanitized) failed on {os.path.basename(src)}")
        r = subprocess.run([nvcc, *ARCH, "-shared", *_SAN, "-o", out, *objs, "-lcudart"], capture_output=True, text=True)
        if r.returncode:
            sys.stderr.write(r.stdout + r.stderr)
            raise RuntimeError("link (sanitized) failed")
    return out


if __name__ == "__main__":
    if "--sanitize" in sys.argv:
        print(build_sanitized())
    else:
        print(build(verbose="--verbose" in sys.argv, force="--force" in sys.argv))
