"""Build the engine's shared libraries in-tree.

``build_cuda()`` compiles the product library ``profess_b200/_lib/libprofess_b200.so``
for sm_100a with nvcc.  ``build_emu()`` compiles the same block functions for
the host into ``tests/_emu/libprofess_b200_emu.so``, a test harness that runs
each CUDA block with one thread so the CPU test suite can check the kernels'
logic against the oracle; the product never loads it.

Usage: python -m profess_b200.build [cuda|emu|all]
"""
from __future__ import annotations

import concurrent.futures
import os
import subprocess
import sys
import tempfile

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
CSRC = os.path.join(HERE, "csrc")
INCLUDE = os.path.join(ROOT, "include")
LIB_DIR = os.path.join(HERE, "_lib")
EMU_DIR = os.path.join(ROOT, "tests", "_emu")
LIB_PATH = os.path.join(LIB_DIR, "libprofess_b200.so")
EMU_PATH = os.path.join(EMU_DIR, "libprofess_b200_emu.so")

# engine.cu and, one unit per pass and precision, the pass kernels
PASS_UNITS = ["pass_%s_%s.cu" % (p, t) for t in ("f64", "f32") for p in ("yzg", "yz", "split", "xfwd", "xinv")]
SOURCES = ["engine.cu"] + PASS_UNITS
HEADERS = ["%s.cuh" % h for h in ("kernels", "cx", "dft", "fft", "dcsrch", "slot", "ntn_ctl", "pass_common", "passes", "setup",
                                  "ewald", "stress")] + [
    "f32/%s.cuh" % h for h in ("kernels", "instantiate", "async", "fft", "shape", "passes")]
# the host emulation: engine.cu takes the FP64 block functions from the headers
EMU_SOURCES = ["engine.cu"] + [u for u in PASS_UNITS if u.endswith("_f32.cu")]

NVCC_FLAGS = [
    "-O3", "-std=c++17", "-lineinfo",
    "-gencode", "arch=compute_100a,code=sm_100a",
    "-Xcompiler", "-fPIC",
    "--expt-relaxed-constexpr",
    "-Xcompiler", "-fopenmp",
]


def _nvcc() -> str:
    for cand in (os.environ.get("NVCC"), "/usr/local/cuda/bin/nvcc", "nvcc"):
        if cand and (os.path.sep not in cand or os.path.exists(cand)):
            return cand
    return "nvcc"


def _stale(target: str) -> bool:
    if not os.path.exists(target):
        return True
    t = os.path.getmtime(target)
    deps = [os.path.join(CSRC, f) for f in SOURCES + HEADERS if os.path.exists(os.path.join(CSRC, f))]
    deps.append(os.path.join(INCLUDE, "profess_b200.h"))
    return any(os.path.getmtime(d) > t for d in deps)


def build_cuda(force: bool = False, extra=None, lib: str = LIB_PATH, csrc: str = CSRC, log: str | None = None) -> str:
    """Compile the units side by side and link them into ``lib`` (``extra``:
    more nvcc flags; ``log``: a file for the compilers' output)."""
    if not force and not _stale(lib):
        return lib
    os.makedirs(os.path.dirname(lib), exist_ok=True)
    tmp = tempfile.TemporaryDirectory()
    objs = [os.path.join(tmp.name, s[:-3] + ".o") for s in SOURCES]

    def compile_unit(src, obj):
        cmd = [_nvcc()] + NVCC_FLAGS + (extra or []) + ["-I", INCLUDE, "-I", csrc, "-c", os.path.join(csrc, src), "-o", obj]
        r = subprocess.run(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)
        if r.returncode:
            raise RuntimeError("%s\n%s" % (" ".join(cmd), r.stdout))
        return r.stdout

    with concurrent.futures.ThreadPoolExecutor(max_workers=os.cpu_count() or 1) as pool:
        out = list(pool.map(compile_unit, SOURCES, objs))
    if log:
        with open(log, "w") as fh:
            fh.write("".join(out))
    subprocess.run([_nvcc(), "-shared", "-gencode", "arch=compute_100a,code=sm_100a", "-Xcompiler", "-fopenmp"] + objs +
                   ["-lgomp", "-o", lib], check=True)
    tmp.cleanup()
    return lib


def build_emu(force: bool = False) -> str:
    if not force and not _stale(EMU_PATH):
        return EMU_PATH
    os.makedirs(EMU_DIR, exist_ok=True)
    cmd = ["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-fopenmp", "-DOFDFT_EMU", "-x", "c++",
           "-I", INCLUDE, "-I", CSRC] + [os.path.join(CSRC, s) for s in EMU_SOURCES] + ["-o", EMU_PATH]
    subprocess.run(cmd, check=True)
    return EMU_PATH


if __name__ == "__main__":
    what = sys.argv[1] if len(sys.argv) > 1 else "all"
    if what in ("cuda", "all"):
        print(build_cuda(force=True))
    if what in ("emu", "all"):
        print(build_emu(force=True))
