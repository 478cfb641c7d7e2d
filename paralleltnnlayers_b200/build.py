"""Build libb200cp.so in-tree with nvcc for sm_100a, and the torch binding over it.

    python -m paralleltnnlayers_b200.build [--force] [--verbose]

Each .cu under csrc/ is compiled to an object (rebuilt only when it or a header it includes
is newer) and linked into ``paralleltnnlayers_b200/libb200cp.so``.  The library
has no dependency on torch; it links the CUDA runtime and NCCL only.  The one
.cpp file there is the CPython / torch binding, ``paralleltnnlayers_b200/_C.so``,
which links the library (found next to it) and is imported after torch.
"""
from __future__ import annotations

import glob
import os
import re
import subprocess
import sys
from concurrent.futures import ThreadPoolExecutor

PKG = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(PKG)
CSRC = os.path.join(PKG, "csrc")
OBJ = os.path.join(PKG, "csrc", "_obj")
LIB = os.path.join(PKG, "libb200cp.so")
BINDING = os.path.join(PKG, "_C.so")

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
    "-Xcompiler", "-fPIC", "-Xcompiler", "-fvisibility=hidden", "--expt-relaxed-constexpr",
    "-I", os.path.join(ROOT, "include"), "-I", CSRC,
]


# extra nvcc flags for experiments, e.g. B200CP_NVCC_FLAGS="-DB200CP_TRACE" (forces nothing by itself: use --force)
NVCC_FLAGS += os.environ.get("B200CP_NVCC_FLAGS", "").split()


def _newest_source(path, seen=None):
    """Modification time of the newest of a source and the project headers it includes, directly or through others."""
    seen = set() if seen is None else seen
    seen.add(path)
    t = os.path.getmtime(path)
    with open(path) as f:
        names = re.findall(r'^\s*#\s*include\s+"([^"]+)"', f.read(), re.M)
    for n in names:
        for d in (os.path.dirname(path), CSRC, os.path.join(ROOT, "include")):
            h = os.path.join(d, n)
            if os.path.exists(h):
                if h not in seen:
                    t = max(t, _newest_source(h, seen))
                break
    return t


def _compile(src, force, verbose):
    obj = os.path.join(OBJ, os.path.basename(src)[:-3] + ".o")
    if not force and os.path.exists(obj) and os.path.getmtime(obj) > _newest_source(src):
        return obj, False
    cmd = ["nvcc", "-c", src, "-o", obj] + NVCC_FLAGS + (["-Xptxas", "-v"] if verbose else [])
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError(f"nvcc failed for {src}:\n{r.stdout}\n{r.stderr}")
    if verbose:
        sys.stderr.write(r.stderr)
    return obj, True


def build(force=False, verbose=False):
    os.makedirs(OBJ, exist_ok=True)
    srcs = sorted(glob.glob(os.path.join(CSRC, "*.cu")))
    with ThreadPoolExecutor(max_workers=min(8, len(srcs))) as ex:
        res = list(ex.map(lambda s: _compile(s, force, verbose), srcs))
    objs = [o for o, _ in res]
    if force or any(ch for _, ch in res) or not os.path.exists(LIB):
        cmd = ["nvcc", "-shared", "-o", LIB] + objs + ["-gencode", "arch=compute_100a,code=sm_100a",
                                                     "-Xcompiler", "-fPIC", "-lcudart"]
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode != 0:
            raise RuntimeError(f"link failed:\n{r.stdout}\n{r.stderr}")
    _build_binding(force)
    return LIB


def _build_binding(force):
    src = os.path.join(CSRC, "torch_binding.cpp")
    hdr = os.path.join(ROOT, "include", "b200cp.h")
    if not force and os.path.exists(BINDING) and os.path.getmtime(BINDING) > max(os.path.getmtime(src), os.path.getmtime(hdr)):
        return
    import sysconfig

    import torch
    tdir = os.path.dirname(torch.__file__)
    inc = [os.path.join(ROOT, "include"), os.path.join(tdir, "include"),
           os.path.join(tdir, "include", "torch", "csrc", "api", "include"), sysconfig.get_paths()["include"],
           "/usr/local/cuda/include"]
    cmd = ["g++", "-shared", "-fPIC", "-O2", "-std=c++17", "-fvisibility=hidden", "-Wno-deprecated-declarations",
           f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}", src, "-o", BINDING]
    cmd += [f for i in inc for f in ("-isystem" if i != inc[0] else "-I", i)]
    cmd += ["-L" + os.path.join(tdir, "lib"), "-L" + PKG, "-l:libb200cp.so", "-ltorch_python", "-ltorch", "-ltorch_cpu",
            "-ltorch_cuda", "-lc10", "-lc10_cuda", "-Wl,-rpath,$ORIGIN"]
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError(f"the torch binding did not build:\n{r.stdout}\n{r.stderr}")


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="--verbose" in sys.argv))
