"""Ahead-of-time build of ``libpx_b200.so`` (sm_100a only) with nvcc; no GPU is needed to build."""
from __future__ import annotations

import os
import shutil
import subprocess
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
LIB = os.path.join(HERE, "libpx_b200.so")
EXT_SRC = os.path.join(CSRC, "torch_ext.cpp")       # the native host path: C++ only, built against torch's headers
EXT = os.path.join(HERE, "_C.so")
SOURCES = ["api.cu", "layer_norm.cu", "trimul.cu", "trimul_in_tc.cu", "trimul_out_tc.cu", "contract_tcgen05.cu", "flash_tcgen05.cu", "triatt.cu", "triatt_in_tc.cu", "triatt_out_tc.cu", "pair_bias_tc.cu", "recycle_tc.cu", "transition_tcgen05.cu", "peer.cu", "selftest.cu", "standardise.cu", "opm_tc.cu", "dropout_add.cu", "single_tc.cu", "msa_rows_tc.cu", "msa_transition_tc.cu",
           "msa_average_tc.cu", "msa_embed.cu"]
NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17", "-lineinfo",
    "--expt-relaxed-constexpr", "-Xcompiler", "-fPIC", "-Xcompiler", "-fvisibility=hidden",
]


def _nvcc() -> str:
    for cand in (os.environ.get("NVCC"), shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if cand and os.path.exists(cand):
            return cand
    raise RuntimeError("nvcc not found: libpx_b200.so cannot be built")


def needs_build() -> bool:
    if not os.path.exists(LIB):
        return True
    t = os.path.getmtime(LIB)
    deps = [os.path.join(CSRC, f) for f in os.listdir(CSRC) if not f.endswith(".cpp")] + [os.path.join(HERE, "..", "include", "px_b200.h")]
    return any(os.path.getmtime(d) > t for d in deps)


def build_ext(force: bool = False) -> str:
    """Compile csrc/torch_ext.cpp into ``_C.so`` next to this file."""
    import sysconfig

    import torch

    deps = [EXT_SRC, os.path.join(HERE, "..", "include", "px_b200.h")]
    if not force and os.path.exists(EXT) and all(os.path.getmtime(d) <= os.path.getmtime(EXT) for d in deps):
        return EXT
    root = os.path.dirname(torch.__file__)
    cuda = os.path.dirname(os.path.dirname(_nvcc()))
    inc = [sysconfig.get_paths()["include"], os.path.join(root, "include"),
           os.path.join(root, "include", "torch", "csrc", "api", "include"), os.path.join(cuda, "include")]
    cmd = [os.environ.get("CXX", "g++"), "-std=c++17", "-O2", "-fPIC", "-fvisibility=hidden", "-Wno-interference-size", "-shared", EXT_SRC, "-o", EXT,
           *["-I" + d for d in inc], "-L" + os.path.join(root, "lib"), "-L" + os.path.join(cuda, "lib64"),
           "-lc10", "-lc10_cuda", "-ltorch_cpu", "-ltorch_cuda", "-ltorch", "-ltorch_python",
           f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}"]
    subprocess.check_call(cmd)
    return EXT


def build(force: bool = False, verbose: bool = False) -> str:
    """Compile every .cu under csrc/ into one shared library next to this file, and the host path beside it."""
    build_ext(force)
    if not force and not needs_build():
        return LIB
    objdir = os.path.join(HERE, "build")
    os.makedirs(objdir, exist_ok=True)
    nvcc = _nvcc()
    procs = []
    for src in SOURCES:
        obj = os.path.join(objdir, src.replace(".cu", ".o"))
        cmd = [nvcc, *NVCC_FLAGS, "-c", os.path.join(CSRC, src), "-o", obj]
        if verbose:
            cmd.insert(1, "-Xptxas")
            cmd.insert(2, "-v")
        procs.append((src, obj, subprocess.Popen(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)))
    objs = []
    for src, obj, p in procs:
        out, _ = p.communicate()
        if verbose or p.returncode != 0:
            sys.stderr.write(out)
        if p.returncode != 0:
            raise RuntimeError(f"nvcc failed on {src}")
        objs.append(obj)
    cmd = [nvcc, "-shared", "-o", LIB, *objs, "-gencode", "arch=compute_100a,code=sm_100a"]
    subprocess.check_call(cmd)
    return LIB


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))
