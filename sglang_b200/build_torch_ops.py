"""Build the two host-only libraries over the C ABI of ``libsglb200.so`` that need torch's headers:

* ``sglang_b200/lib/libsgl_kernel_ops.so``: the torch registration of the ``sgl_kernel`` ops on this path
  (``TORCH_LIBRARY_FRAGMENT(sgl_kernel, m)``, schemas of ``sgl-kernel/csrc/common_extension.cc``);
  ``sglang_b200.sgl_kernel.load_torch_ops()`` loads it, after which the ops are reachable as
  ``torch.ops.sgl_kernel.<name>`` like the reference's;
* ``sglang_b200/lib/_sglb200_host.so``: the compiled host path of the layer-level functions (a CPython module).

    python -m sglang_b200.build_torch_ops [--force]

One translation unit each, compiled with g++ against the installed torch headers and linked to ``libsglb200.so``
through ``$ORIGIN``; no kernel lives in them.
"""

from __future__ import annotations

import argparse
import os
import shutil
import subprocess
import sys
import sysconfig
from concurrent.futures import ThreadPoolExecutor

PKG = os.path.dirname(os.path.abspath(__file__))
SRCDIR = os.path.join(PKG, "csrc", "torch_ops")
LIBDIR = os.path.join(PKG, "lib")
OUT = os.path.join(LIBDIR, "libsgl_kernel_ops.so")
HOST = os.path.join(LIBDIR, "_sglb200_host.so")


def _compile(src: str, out: str, extra_incs, extra_libs, force: bool) -> str:
    import torch
    from torch.utils.cpp_extension import include_paths
    hdr = os.path.join(os.path.dirname(PKG), "include", "sglb200.h")
    # the core library only has to exist: what is compiled in here is its header
    newest = max(os.path.getmtime(p) for p in (src, hdr))
    if not force and os.path.exists(out) and os.path.getmtime(out) >= newest:
        return out
    cxx = os.environ.get("CXX") or shutil.which("g++")
    if not cxx:
        raise RuntimeError(f"g++ not found: cannot build {os.path.basename(out)}")
    tlib = os.path.join(os.path.dirname(torch.__file__), "lib")
    cuda_home = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    incs = include_paths() + [os.path.join(cuda_home, "include"), *extra_incs]
    tmp = f"{out}.{os.getpid()}.tmp"
    cmd = [cxx, "-O2", "-std=c++17", "-fPIC", "-shared", "-Wno-deprecated-declarations",
           f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
           *[f"-I{i}" for i in incs], src, "-o", tmp,
           f"-L{tlib}", "-lc10", "-lc10_cuda", "-ltorch_cpu", "-ltorch_cuda", "-ltorch", *extra_libs,
           f"-L{LIBDIR}", "-lsglb200", "-Wl,-rpath,$ORIGIN", f"-Wl,-rpath,{tlib}"]
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        sys.stderr.write(r.stdout + r.stderr)
        if os.path.exists(tmp):
            os.remove(tmp)
        raise RuntimeError(f"build of {os.path.basename(out)} failed")
    os.replace(tmp, out)
    return out


def build(force: bool = False) -> str:
    from . import build as base
    base.build()
    jobs = [(os.path.join(SRCDIR, "sgl_kernel_ops.cpp"), OUT, [], [], force),
            (os.path.join(SRCDIR, "host_path.cpp"), HOST, [sysconfig.get_paths()["include"]], ["-ltorch_python"], force)]
    with ThreadPoolExecutor(max_workers=2) as ex:
        list(ex.map(lambda j: _compile(*j), jobs))
    return OUT


if __name__ == "__main__":
    ap = argparse.ArgumentParser()
    ap.add_argument("--force", action="store_true")
    print(build(ap.parse_args().force))
