"""Build step of the C-ABI library: nvcc for sm_100a only, in-tree output.

``python lightop_b200/build.py`` (run by path: importing the package needs the built library) compiles ``csrc/*.cu`` into
``lightop_b200/liblightop_b200.so`` and, where a torch with CUDA is installed, ``csrc/host.cpp`` (the host side of small calls, against that
torch) into ``lightop_b200/_host.so``.  nvcc cross-compiles without a GPU.
"""
from __future__ import annotations

import importlib.util
import os
import runpy
import subprocess
import sys
import sysconfig

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
LIB = os.path.join(HERE, "liblightop_b200.so")
HOST = os.path.join(HERE, "_host.so")
SOURCES = ["common.cu", "quant.cu", "routing.cu", "gate.cu", "reduce.cu", "grouped_gemm.cu", "fused_moe.cu", "grouped_layouts.cu", "peer.cu"]
NVCC_FLAGS = ["-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17", "-lineinfo",
              "-Xcompiler", "-fPIC", "--expt-relaxed-constexpr"]


def _nvcc() -> str:
    for cand in (os.environ.get("NVCC"), "/usr/local/cuda/bin/nvcc", "nvcc"):
        if cand and (os.path.isabs(cand) and os.path.exists(cand) or not os.path.isabs(cand)):
            return cand
    return "nvcc"


def _dependencies(out: str) -> list:
    """The sources of an output (the object files that a build leaves beside them are none: they are newer than an output that was linked first)."""
    headers = [os.path.join(HERE, "..", "include", "lightop_b200.h")]
    if out == HOST:
        return [os.path.join(CSRC, "host.cpp"), *headers]
    return [*(os.path.join(CSRC, f) for f in SOURCES), *(os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith(".h")), *headers]


def _torch_dir() -> str:
    """Where the installed torch is, "" if there is none (found without importing it: a first import takes a while)."""
    spec = importlib.util.find_spec("torch")
    return list(spec.submodule_search_locations)[0] if spec is not None and spec.submodule_search_locations else ""


def host_possible() -> bool:
    """Whether there is a torch with CUDA to compile the host module against.  The C-ABI library needs none, and the package goes without the module."""
    torch_dir = _torch_dir()
    return bool(torch_dir) and os.path.exists(os.path.join(torch_dir, "lib", "libc10_cuda.so"))


def built_for() -> str:
    """What the host module is compiled against besides its sources; it carries this text, and one with another text is out of date."""
    torch_version = runpy.run_path(os.path.join(_torch_dir(), "version.py"))["__version__"]
    return f"torch {torch_version}, Python {sysconfig.get_config_var('SOABI')}"


def _host_marker() -> bytes:
    return f"[built for {built_for()}]".encode()


def outdated() -> list:
    """The outputs, of LIB and HOST, that are missing, older than one of their sources or (HOST) built for another torch or Python."""
    def old(out):
        if not os.path.exists(out):
            return True
        if out == HOST:
            with open(out, "rb") as f:
                if _host_marker() not in f.read():
                    return True
        t = os.path.getmtime(out)
        return any(os.path.getmtime(d) > t for d in _dependencies(out))
    return [out for out in _outputs() if old(out)]


def _outputs() -> list:
    return [LIB, HOST] if host_possible() else [LIB]


def needs_build() -> bool:
    return bool(outdated())


def _host_command(out: str) -> list:
    torch_dir = _torch_dir()
    cuda_dir = os.path.dirname(os.path.dirname(_nvcc())) if os.path.isabs(_nvcc()) else "/usr/local/cuda"
    include = [os.path.join(torch_dir, "include"), os.path.join(torch_dir, "include", "torch", "csrc", "api", "include"),
               os.path.join(cuda_dir, "include"), sysconfig.get_path("include")]
    lib = os.path.join(torch_dir, "lib")
    return [os.environ.get("CXX", "g++"), "-O2", "-std=c++17", "-fPIC", "-shared", f'-DLIGHTOP_BUILT_FOR="{_host_marker().decode()}"', *[f"-I{d}" for d in include], os.path.join(CSRC, "host.cpp"),
            "-o", out, f"-L{lib}", "-lc10", "-lc10_cuda", "-ltorch_cpu", "-ltorch_python", f"-Wl,-rpath,{lib}"]


def _compile(commands: list, verbose: bool = False) -> None:
    """Runs (source, command) pairs side by side."""
    procs = [(src, subprocess.Popen(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)) for src, cmd in commands]
    results = [(src, pr.communicate()[0], pr.returncode) for src, pr in procs]
    for src, out, rc in results:
        if rc != 0:
            raise RuntimeError(f"the compiler failed on {src}:\n{out}")
        if verbose and out:
            print(out)


def build(force: bool = False, verbose: bool = False) -> str:
    todo = _outputs() if force else outdated()
    # An output is written under another name and renamed when it is complete: a process that has the old file mapped keeps it, and a build that
    # fails leaves it.
    part = {out: f"{out[:-len('.so')]}.{os.getpid()}.so" for out in todo}
    try:
        if LIB in todo:
            objs = [os.path.join(CSRC, src.replace(".cu", ".o")) for src in SOURCES]
            _compile([(src, [_nvcc(), *(["-Xptxas=-v"] if verbose else []), *NVCC_FLAGS, "-c", os.path.join(CSRC, src), "-o", obj])
                      for src, obj in zip(SOURCES, objs)], verbose)
            res = subprocess.run([_nvcc(), "-shared", "-o", part[LIB], *objs, "-cudart", "static"], stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)
            if res.returncode != 0:
                raise RuntimeError(f"link failed:\n{res.stdout}")
            os.replace(part[LIB], LIB)
        if HOST in todo:      # last: where it does not compile, the library is there and the package works without it
            _compile([("host.cpp", _host_command(part[HOST]))], verbose)
            os.replace(part[HOST], HOST)
    finally:
        for path in part.values():
            if os.path.exists(path):
                os.unlink(path)
    return LIB


def build_tools(force: bool = False) -> str:
    """Compile the stand-alone MMA-peak micro-benchmark next to bench.py, which runs it for the INT8 tensor peak."""
    root = os.path.dirname(HERE)
    src = os.path.join(root, "bench_mma_peak.cu")
    exe = os.path.join(root, "bench_mma_peak")
    if force or not os.path.exists(exe) or os.path.getmtime(src) > os.path.getmtime(exe):
        res = subprocess.run([_nvcc(), "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-lineinfo", "-o", exe, src],
                             stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)
        if res.returncode != 0:
            raise RuntimeError(f"nvcc failed on bench_mma_peak.cu:\n{res.stdout}")
    return exe


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))
    if "--tools" in sys.argv:
        print(build_tools(force="--force" in sys.argv))
