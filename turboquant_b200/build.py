"""Builds libturboquant_b200.so (the C-ABI library) in-tree with nvcc for sm_100a, and the native call path of the
Python layer (_native.so, the one file that sees torch's headers) with g++.

    python -m turboquant_b200.build [--force]

The cache-write, flat-quantizer and bulk-dequantizer translation units are compiled with -fmad=false: their
arithmetic must round every product and sum separately to stay bit-identical to the torch
quantizer.  The library itself involves no torch headers and exports plain C symbols only.
"""
from __future__ import annotations

import shutil
import subprocess
import sys
from concurrent.futures import ThreadPoolExecutor
from pathlib import Path

PKG = Path(__file__).resolve().parent
CSRC = PKG / "csrc"
LIB_DIR = PKG / "lib"
LIB = LIB_DIR / "libturboquant_b200.so"
NATIVE = PKG / "_native.so"
NATIVE_SRC = CSRC / "tq_torch.cpp"
NATIVE_STAMP = PKG / "build" / "native.stamp"      # what NATIVE was built against
HEADER = PKG.parent / "include" / "turboquant_b200.h"

ARCH = ["-gencode", "arch=compute_100a,code=sm_100a"]
COMMON = ["-O3", "-std=c++17", "-lineinfo", "-Xcompiler", "-fPIC", "--expt-relaxed-constexpr"]
UNITS = {
    "tq_api.cu": [],
    "tq_write.cu": ["-fmad=false"],
    "tq_write_rows.cu": ["-fmad=false"],
    "tq_flat.cu": ["-fmad=false"],
    "tq_flat_rows.cu": ["-fmad=false"],
    "tq_flat_quant.cu": ["-fmad=false"],
    "tq_decode.cu": [],
    "tq_decode_mq.cu": [],
    "tq_decode_split.cu": [],
    "tq_dequant.cu": ["-fmad=false"],
    "tq_pages.cu": [],
    "tq_generic.cu": ["-fmad=false"],
    "tq_nc.cu": ["-fmad=false"],
}


def _stale(target: Path, sources) -> bool:
    if not target.exists():
        return True
    t = target.stat().st_mtime
    return any(Path(s).stat().st_mtime > t for s in sources)


def _native_command() -> list[str]:
    import sysconfig
    import torch
    root = Path(torch.__file__).resolve().parent
    cuda = Path(shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc").resolve().parent.parent
    return ["g++", "-O2", "-std=c++17", "-fPIC", "-shared", f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
            "-isystem", str(root / "include"), "-isystem", str(root / "include/torch/csrc/api/include"),
            "-I", str(cuda / "include"), "-I", sysconfig.get_paths()["include"], str(NATIVE_SRC), "-o", str(NATIVE),
            "-L", str(root / "lib"), "-lc10", "-lc10_cuda", "-ltorch_cpu", "-ltorch_python"]


def _native_stamp() -> str:
    import sysconfig
    import torch
    return "\n".join([torch.__version__, str(sysconfig.get_config_var("SOABI")), *_native_command()])


def _native_stale() -> bool:
    """Older than its source, or built against another torch or Python: the module is bound to both."""
    built_against = NATIVE_STAMP.read_text() if NATIVE_STAMP.exists() else ""
    return _stale(NATIVE, [NATIVE_SRC, HEADER, Path(__file__)]) or built_against != _native_stamp()


def _build_native() -> None:
    subprocess.check_call(_native_command())
    NATIVE_STAMP.write_text(_native_stamp())


def build(force: bool = False, verbose: bool = False) -> Path:
    LIB_DIR.mkdir(exist_ok=True)
    obj_dir = PKG / "build"
    obj_dir.mkdir(exist_ok=True)
    deps = [CSRC / "tq_common.cuh", CSRC / "tq_rows.cuh", CSRC / "tq_decode_common.cuh", HEADER, Path(__file__)]

    def compile_one(item):
        name, extra = item
        src, obj = CSRC / name, obj_dir / (name + ".o")
        if force or _stale(obj, [src, *deps]):
            cmd = ["nvcc", *ARCH, *COMMON, *extra, "-c", str(src), "-o", str(obj)]
            if verbose:
                cmd.insert(1, "-Xptxas=-v")
                print(" ".join(cmd), flush=True)
            subprocess.check_call(cmd)
        return obj

    with ThreadPoolExecutor(max_workers=5) as ex:
        native = None
        if force or _native_stale():
            native = ex.submit(_build_native)
        objs = list(ex.map(compile_one, UNITS.items()))
        if native:
            native.result()
    if force or _stale(LIB, objs):
        subprocess.check_call(["nvcc", *ARCH, "-shared", "-o", str(LIB), *map(str, objs)])
    return LIB


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))
