"""Build libgint_b200.so (the CUDA kernels + C ABI) in-tree with nvcc for sm_100a.

    python -m gint_b200.build [--force] [--jobs N] [--no-hot-order] [-D MACRO=VALUE ...]

Pipeline, per interpreter kernel in ``gint_b200/csrc/kernels/*.cu``:

    nvcc -cubin                    CUDA C++ with inline PTX -> sm_100a machine code
    .incbin                        the cubin becomes a byte array in an object file

then ``gint_capi.cu`` (host code) is compiled and everything is linked into ``gint_b200/libgint_b200.so`` with the CUDA
runtime linked statically. nvcc cross-compiles without a GPU, so this also runs on a CPU-only machine. A unit is rebuilt
when its source, a header that it includes (listed in a .d file by its last build) or this file is newer than its output.
"""
from __future__ import annotations

import argparse
import concurrent.futures
import glob
import os
import shutil
import subprocess
import sys
import time

PKG_DIR = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(PKG_DIR, "csrc")
KERNELS = os.path.join(CSRC, "kernels")
OBJ_DIR = os.path.join(CSRC, "build")
HOT_HEADER = os.path.join(OBJ_DIR, "gint_hot_handlers.h")
LANE_HEADER = os.path.join(OBJ_DIR, "gint_lane_programs.h")
LANE_PROGRAMS = ("bmm4x4", "inv4x4")
LIB_PATH = os.path.join(PKG_DIR, "libgint_b200.so")

ARCH = ["-gencode", "arch=compute_100a,code=sm_100a"]
COMMON = ["-lineinfo", "-O3", "-std=c++17",
          "-fmad=false", "--diag-suppress", "20013"]   # the bytecode's FMul/FAdd must stay separate roundings; FMA is its own opcode


def _nvcc() -> str:
    exe = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(exe):
        raise RuntimeError("nvcc not found; cannot build libgint_b200.so")
    return exe


STEP_TIMEOUT_S = 900    # a compiler step that runs this long is stuck (ptxas on an unlucky control-flow graph): fail, do not hang


def _run(cmd: list[str], what: str) -> str:
    try:
        r = subprocess.run(cmd, capture_output=True, text=True, timeout=STEP_TIMEOUT_S)
    except subprocess.TimeoutExpired:
        raise RuntimeError(f"{what} did not finish within {STEP_TIMEOUT_S} s:\n{' '.join(cmd)}")
    if r.returncode != 0:
        raise RuntimeError(f"{what} failed:\n{' '.join(cmd)}\n{r.stdout}\n{r.stderr}")
    return r.stderr + r.stdout


def _outdated(obj: str) -> bool:
    """Is a file that `obj` was made from (its .d file) newer than it, or not known?"""
    dep = obj[:-2] + ".d"
    if not os.path.exists(obj) or not os.path.exists(dep):
        return True
    with open(dep) as f:
        files = f.read().split(":", 1)[1].replace("\\\n", " ").split()
    made = os.path.getmtime(obj)
    return any(not os.path.exists(h) or os.path.getmtime(h) > made for h in files + [__file__])


def _write_hot_header(ordered: bool) -> None:
    """The handlers that come first in the kernels' code (hot_handlers.json) as macro lists X(opcode, stack depth), one per kernel family."""
    from . import hot_handlers
    text = "/* written by gint_b200/build.py from hot_handlers.json */\n"
    for family in ("plain", "rf", "vec"):
        keys = sorted(hot_handlers.load(family)) if ordered else []
        text += f"#define GINT_HOT_{family.upper()}(X) " + " ".join(f"X({op}, {depth})" for depth, op in keys) + "\n"
    if not os.path.exists(HOT_HEADER) or open(HOT_HEADER).read() != text:
        with open(HOT_HEADER, "w") as f:
            f.write(text)


def _write_lane_header() -> None:
    """The small-matrix programs that get a kernel of their own (gint_lanes.cuh), as constant tables: the recorded streams, which do not
    depend on the batch size."""
    import json
    with open(os.path.join(PKG_DIR, "data", "programs.json")) as f:
        records = json.load(f)
    text = "/* written by gint_b200/build.py from data/programs.json */\n#pragma once\nnamespace gint {\n"
    for name in LANE_PROGRAMS:
        code = [v for pair in records[name + "_b1"]["bytecode"] for v in (pair if isinstance(pair, list) else [pair])]
        pairs = list(zip(code[::2], code[1::2]))
        text += f"struct LaneCode_{name} {{\n    static constexpr int n = {len(pairs)};\n    static constexpr int code[{len(pairs)}][2] = {{" + \
            ", ".join(f"{{{op}, {arg}}}" for op, arg in pairs) + "};\n};\n"
    text += "}  // namespace gint\n#define GINT_LANE_PROGRAMS(X) " + " ".join(f"X({name})" for name in LANE_PROGRAMS) + "\n"
    if not os.path.exists(LANE_HEADER) or open(LANE_HEADER).read() != text:
        with open(LANE_HEADER, "w") as f:
            f.write(text)


def _build_kernel(src: str, extra: list[str]) -> tuple[str, str]:
    """CUDA C++ -> cubin -> object with the cubin as a byte array."""
    stem = os.path.basename(src)[:-3]                       # gint_direct_p4_k1
    sym = stem.replace("gint_", "gint_cubin_").replace("_p", "_").replace("_k", "_")   # gint_cubin_direct_4_1
    cubin, obj = (os.path.join(OBJ_DIR, stem + ext) for ext in (".cubin", ".o"))
    t0 = time.time()
    log = _run([_nvcc(), "-arch=sm_100a", "-cubin", "-Xptxas", "-v", "-I", OBJ_DIR, "-MD", "-MF", obj[:-2] + ".d"] + COMMON + extra + [src, "-o", cubin], f"nvcc {stem}")
    log += f"build time: {time.time() - t0:.0f} s\n"
    asm = os.path.join(OBJ_DIR, stem + ".S")
    with open(asm, "w") as f:
        f.write(f'.section .rodata\n.balign 64\n.global {sym}\n{sym}:\n.incbin "{cubin}"\n.global {sym}_end\n{sym}_end:\n.byte 0\n'
                '.section .note.GNU-stack,"",@progbits\n')
    _run(["gcc", "-c", asm, "-o", obj], f"as {stem}")
    return stem, log


def build(force: bool = False, jobs: int | None = None, verbose: bool = False, extra_flags: list[str] | None = None,
          hot_order: bool = True) -> str:
    os.makedirs(OBJ_DIR, exist_ok=True)
    extra = list(extra_flags or [])
    stamp = os.path.join(OBJ_DIR, "flags.txt")
    flags_now = " ".join(extra) + f" hot_order={hot_order}"
    if not os.path.exists(stamp) or open(stamp).read() != flags_now:
        force = True
    _write_hot_header(hot_order)
    _write_lane_header()
    kernels = sorted(glob.glob(os.path.join(KERNELS, "*.cu")))
    todo, objs = [], []
    for src in kernels:
        obj = os.path.join(OBJ_DIR, os.path.basename(src)[:-3] + ".o")
        objs.append(obj)
        if force or _outdated(obj):
            todo.append(src)
    logs = []
    capi_src = os.path.join(CSRC, "gint_capi.cu")
    capi_obj = os.path.join(OBJ_DIR, "gint_capi.o")
    objs.append(capi_obj)
    capi_todo = force or _outdated(capi_obj)
    with concurrent.futures.ThreadPoolExecutor(max_workers=jobs or os.cpu_count() or 4) as ex:
        futs = [ex.submit(_build_kernel, s, extra) for s in todo]
        if capi_todo:
            futs.append(ex.submit(lambda: ("gint_capi", _run([_nvcc()] + ARCH + COMMON + ["-I", OBJ_DIR, "-Xcompiler", "-fPIC", "-MD", "-MF", capi_obj[:-2] + ".d", "-c", capi_src, "-o", capi_obj],
                                                              "nvcc gint_capi"))))
        for f in concurrent.futures.as_completed(futs):
            logs.append(f.result())
    if todo or capi_todo or not os.path.exists(LIB_PATH):
        _run([_nvcc(), "-shared", "-o", LIB_PATH] + objs, "link")
    with open(stamp, "w") as f:
        f.write(flags_now)
    if verbose:
        for name, log in sorted(logs):
            for line in log.splitlines():
                if "registers" in line or "build time" in line or ("spill" in line and "0 bytes spill stores" not in line):
                    print(f"[{name}] {line.strip()}")
    return LIB_PATH


def main() -> None:
    ap = argparse.ArgumentParser()
    ap.add_argument("--force", action="store_true")
    ap.add_argument("--jobs", type=int, default=None)
    ap.add_argument("--no-hot-order", action="store_true", help="handlers in plain order, not the recorded programs' first (for A/B measurements)")
    ap.add_argument("-D", dest="defines", action="append", default=[])
    opts = ap.parse_args()
    path = build(force=opts.force, jobs=opts.jobs, verbose=True, extra_flags=[f"-D{d}" for d in opts.defines],
                 hot_order=not opts.no_hot_order)
    print(path)


if __name__ == "__main__":
    sys.exit(main())
