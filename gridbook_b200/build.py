"""Build recipe: libgridbook_b200.so (nvcc, sm_100a only) and the host path _gb_torch.so (g++, against
the installed torch), both in-tree."""
from __future__ import annotations

import hashlib
import os
import shutil
import subprocess
import sys
import sysconfig

PKG = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(PKG, "csrc")
LIB = os.path.join(PKG, "libgridbook_b200.so")
HOST_LIB = os.path.join(PKG, "_gb_torch.so")
HOST_SOURCE = "gb_torch.cpp"
SOURCES = ("gb_api.cu", "gb_decode.cu", "gb_gemv.cu", "gb_moe.cu", "gb_gemm.cu", "gb_gemv_dot.cu", "gb_peer.cu", "gb_gemv_umma.cu", "gb_gemv_tab.cu", "gb_gemm_fp4.cu", "gb_gemm_pair.cu", "gb_gemm_rows.cu", "gb_gemv_fp4.cu")
HEADERS = ("gb_common.cuh", os.path.join("..", "..", "include", "gridbook_b200.h"))
NVCC_FLAGS = (
    "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
    "--expt-relaxed-constexpr", "-Xcompiler", "-fPIC", "-Xcompiler", "-fvisibility=hidden",
    "-Xptxas", "-v",
)


def _nvcc() -> str:
    for cand in (os.environ.get("NVCC"), shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if cand and os.path.exists(cand):
            return cand
    raise RuntimeError("nvcc not found; libgridbook_b200.so cannot be built")


def source_digest() -> str:
    h = hashlib.sha256()
    for name in SOURCES + HEADERS + (HOST_SOURCE,):
        with open(os.path.join(CSRC, name), "rb") as fh:
            h.update(fh.read())
    h.update(" ".join(NVCC_FLAGS).encode())
    return h.hexdigest()[:16]


def _host_command() -> list[str]:
    """g++ line of the host path: torch's headers and libraries, the Python and CUDA headers."""
    import torch
    from torch.utils import cpp_extension
    inc = cpp_extension.include_paths("cuda") + [sysconfig.get_paths()["include"]]
    lib = os.path.join(os.path.dirname(torch.__file__), "lib")
    return ["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-fvisibility=hidden", "-DTORCH_EXTENSION_NAME=_gb_torch",
            "-DTORCH_API_INCLUDE_EXTENSION_H", f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
            *(f"-isystem{d}" for d in inc), os.path.join(CSRC, HOST_SOURCE), "-o", HOST_LIB,
            f"-L{lib}", "-lc10", "-lc10_cuda", "-ltorch", "-ltorch_cpu", "-ltorch_cuda", "-ltorch_python", "-ldl"]


def build(force: bool = False, verbose: bool = False) -> str:
    """Compile every translation unit and link the shared library. Returns its path."""
    stamp = LIB + ".digest"
    digest = source_digest()
    if (not force and os.path.exists(LIB) and os.path.exists(HOST_LIB) and os.path.exists(stamp)
            and open(stamp).read().strip() == digest):
        return LIB
    nvcc = _nvcc()
    objdir = os.path.join(PKG, "build")
    os.makedirs(objdir, exist_ok=True)
    procs = []
    host = subprocess.Popen(_host_command(), stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)
    for src in SOURCES:
        obj = os.path.join(objdir, src.replace(".cu", ".o"))
        cmd = [nvcc, *NVCC_FLAGS, "-c", os.path.join(CSRC, src), "-o", obj]
        procs.append((src, obj, subprocess.Popen(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT,
                                                text=True)))
    objs, log = [], []
    for src, obj, proc in procs:
        out, _ = proc.communicate()
        log.append(f"==== {src}\n{out}")
        if proc.returncode != 0:
            raise RuntimeError(f"nvcc failed on {src}:\n{out}")
        objs.append(obj)
    with open(os.path.join(objdir, "ptxas.log"), "w") as fh:
        fh.write("\n".join(log))
    link = [nvcc, "-shared", "-o", LIB, *objs, "-gencode", "arch=compute_100a,code=sm_100a",
            "-Xcompiler", "-fPIC", "-lcudart"]
    res = subprocess.run(link, capture_output=True, text=True)
    if res.returncode != 0:
        raise RuntimeError(f"link failed:\n{res.stdout}{res.stderr}")
    out, _ = host.communicate()
    if host.returncode != 0:
        raise RuntimeError(f"g++ failed on {HOST_SOURCE}:\n{out}")
    with open(stamp, "w") as fh:
        fh.write(digest)
    if verbose:
        print("\n".join(log))
    return LIB


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))
