"""Builds libmintb.so (nvcc, sm_100a; cross-compiles without a GPU) and the C++ host side _mintb_host.so (g++ against torch) in-tree.

    python -m mint_plus_b200.build [--force] [--verbose]
"""
from __future__ import annotations

import os
import shutil
import subprocess
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
LIB = os.path.join(HERE, "libmintb.so")
SOURCES = ["api.cu", "prep.cu", "attn_simt.cu", "attn_f32.cu", "sgemm.cu", "sgemm_tc.cu", "attn_tc.cu", "attn_tc_bwd.cu", "gemm_tc.cu", "gemm_bwd.cu", "combine.cu", "glue.cu", "embed_loss.cu", "selftest.cu"]
HOST = os.path.join(CSRC, "host")
HOST_LIB = os.path.join(HERE, "_mintb_host.so")
HOST_SOURCES = ["launch.cpp", "ops.cpp", "layer.cpp", "bind.cpp"]
NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17", "-lineinfo",
    "-Xcompiler", "-fPIC", "-Xcompiler", "-fvisibility=hidden", "--expt-relaxed-constexpr",
]


def _nvcc() -> str:
    cand = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(cand):
        raise RuntimeError("nvcc not found: libmintb.so cannot be built")
    return cand


def _stale(lib: str, folders) -> bool:
    if not os.path.exists(lib):
        return True
    t = os.path.getmtime(lib)
    deps = [os.path.join(d, f) for d in folders for f in os.listdir(d) if f.endswith((".cu", ".cuh", ".cpp", ".h"))]
    return any(os.path.getmtime(d) > t for d in deps)


def _compile(jobs, verbose: bool) -> None:
    """Run the compilers of `jobs` = [(source, command)] side by side."""
    procs = [(src, subprocess.Popen(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)) for src, cmd in jobs]
    failed = []
    for src, p in procs:
        out, _ = p.communicate()
        if verbose or p.returncode != 0:
            sys.stderr.write(out)
        if p.returncode != 0:
            failed.append(src)
    if failed:
        raise RuntimeError(f"compilation failed: {', '.join(failed)}")


def _link(cmd, what: str) -> None:
    r = subprocess.run(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)
    if r.returncode != 0:
        sys.stderr.write(r.stdout)
        raise RuntimeError(f"link of {what} failed")


def _host_jobs():
    """(compile jobs, link command) of the host side.  It is an extension module: found by its name in the package folder, with
    libmintb.so beside it."""
    import sysconfig
    import torch
    root = os.path.dirname(torch.__file__)
    cuda = os.path.dirname(os.path.dirname(_nvcc()))
    inc = [os.path.join(root, "include"), os.path.join(root, "include", "torch", "csrc", "api", "include"), os.path.join(cuda, "include"),
           sysconfig.get_paths()["include"]]
    flags = ["-O2", "-std=c++17", "-fPIC", "-fvisibility=hidden", f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
             *[x for d in inc for x in ("-isystem", d)]]
    objs = [os.path.join(HOST, f[:-4] + ".o") for f in HOST_SOURCES]
    jobs = [(f, ["g++", *flags, "-c", os.path.join(HOST, f), "-o", o]) for f, o in zip(HOST_SOURCES, objs)]
    lib = os.path.join(root, "lib")
    link = ["g++", "-shared", "-o", HOST_LIB, *objs, "-L" + HERE, "-l:libmintb.so", "-L" + lib, "-lc10", "-lc10_cuda", "-ltorch", "-ltorch_cpu", "-ltorch_cuda",
            "-ltorch_python", "-Wl,-rpath,$ORIGIN"]
    return jobs, link


def build(force: bool = False, verbose: bool = False) -> str:
    """Compile every .cu under csrc/ into mint_plus_b200/libmintb.so and csrc/host/*.cpp into _mintb_host.so; returns the first one's path."""
    header = os.path.join(HERE, "..", "include")
    new_lib = force or _stale(LIB, [CSRC, header])
    new_host = force or _stale(HOST_LIB, [HOST, header])
    jobs, host_link = _host_jobs() if new_host else ([], None)
    cuda_objs = [os.path.join(CSRC, src[:-3] + ".o") for src in SOURCES]
    if new_lib:
        nvcc = _nvcc()
        opts = ["-Xptxas=-v"] if verbose else []
        jobs += [(src, [nvcc, *opts, *NVCC_FLAGS, "-c", os.path.join(CSRC, src), "-o", obj]) for src, obj in zip(SOURCES, cuda_objs)]
    _compile(jobs, verbose)
    if new_lib:
        _link([_nvcc(), "-shared", "-o", LIB, *cuda_objs, "-gencode", "arch=compute_100a,code=sm_100a", "-Xlinker", "-soname=libmintb.so"], "libmintb.so")
    if new_host:
        _link(host_link, "_mintb_host.so")
    return LIB


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="--verbose" in sys.argv))
