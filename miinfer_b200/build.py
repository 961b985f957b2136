"""Builds the CUDA library (sm_100a) in-tree with nvcc.

`python -m miinfer_b200.build` compiles miinfer_b200/csrc/*.cu into
miinfer_b200/lib/libb200kv.so, and csrc/python/native.cpp (the CPython module under the
Python mirror's launchers) into miinfer_b200/lib/_native.so.  There is no JIT and no fallback: the Python
mirror loads exactly these files and fails loudly when one is missing.
"""
from __future__ import annotations

import os
import subprocess
import sys
from concurrent.futures import ThreadPoolExecutor
from pathlib import Path

ROOT = Path(__file__).resolve().parent
CSRC = ROOT / "csrc"
LIB_DIR = ROOT / "lib"
LIB_PATH = LIB_DIR / "libb200kv.so"
INCLUDE = ROOT.parent / "include"
NATIVE_SRC = CSRC / "python" / "native.cpp"
NATIVE_PATH = LIB_DIR / "_native.so"     # the CPython module under the Python mirror's launchers
NATIVE_STAMP = LIB_DIR / "_native.stamp"

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a",
    "-O3", "-std=c++17", "-lineinfo", "--use_fast_math",
    "-Xcompiler", "-fPIC", "-Xcompiler", "-fvisibility=hidden",
    "-Xptxas", "-v",
]


def _nvcc() -> str:
    for cand in (os.environ.get("NVCC"), "/usr/local/cuda/bin/nvcc", "nvcc"):
        if cand and (os.path.isabs(cand) and os.path.exists(cand) or not os.path.isabs(cand)):
            return cand
    return "nvcc"


def sources() -> list[Path]:
    return sorted(CSRC.glob("*.cu")) + sorted(CSRC.glob("*.cpp"))


def native_stamp() -> str:
    """What the CPython module is bound to besides its source: it does not load, or not safely, under another."""
    import torch

    return f"python {sys.version}\ntorch {torch.__version__} cxx11abi {torch._C._GLIBCXX_USE_CXX11_ABI}\n"


def needs_build() -> bool:
    if not LIB_PATH.exists() or not NATIVE_PATH.exists():
        return True
    if not NATIVE_STAMP.exists() or NATIVE_STAMP.read_text() != native_stamp():
        return True
    newest = max(p.stat().st_mtime for p in list(CSRC.glob("*")) + [NATIVE_SRC, INCLUDE / "b200kv.h"])
    return newest > min(LIB_PATH.stat().st_mtime, NATIVE_PATH.stat().st_mtime)


def native_command() -> list[str]:
    import sysconfig

    import torch
    from torch.utils.cpp_extension import include_paths, library_paths

    cuda = Path(_nvcc()).resolve().parent.parent / "include"
    return ["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-fvisibility=hidden", f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
            f"-I{INCLUDE}", *[f"-isystem{p}" for p in [*include_paths(), sysconfig.get_paths()["include"], str(cuda)]], str(NATIVE_SRC),
            "-o", str(NATIVE_PATH), *[f"-L{p}" for p in library_paths()], "-lc10", "-lc10_cuda", "-ltorch_cpu", "-ltorch_python", "-ltorch"]


def build(force: bool = False, verbose: bool = False) -> Path:
    if not force and not needs_build():
        return LIB_PATH
    LIB_DIR.mkdir(exist_ok=True)
    obj_dir = ROOT / "build"
    obj_dir.mkdir(exist_ok=True)
    nvcc = _nvcc()

    def compile_one(src: Path) -> tuple[Path, str]:
        obj = obj_dir / (src.stem + ".o")
        cmd = [nvcc, *NVCC_FLAGS, f"-I{INCLUDE}", f"-I{CSRC}", "-c", str(src), "-o", str(obj)]
        res = subprocess.run(cmd, capture_output=True, text=True)
        if res.returncode != 0:
            raise RuntimeError(f"nvcc failed for {src.name}:\n{res.stdout}\n{res.stderr}")
        return obj, res.stderr

    def compile_native() -> None:
        res = subprocess.run(native_command(), capture_output=True, text=True)
        if res.returncode != 0:
            raise RuntimeError(f"g++ failed for {NATIVE_SRC.name}:\n{res.stdout}\n{res.stderr}")
        NATIVE_STAMP.write_text(native_stamp())

    with ThreadPoolExecutor(max_workers=min(8, os.cpu_count() or 1)) as pool:
        native = pool.submit(compile_native)
        results = list(pool.map(compile_one, sources()))
        native.result()
    log = "\n".join(f"== {obj.name}\n{err}" for obj, err in results)
    (obj_dir / "ptxas.log").write_text(log)
    if verbose:
        print(log)
    cmd = [nvcc, "-shared", "-gencode", "arch=compute_100a,code=sm_100a", "-o", str(LIB_PATH),
           *[str(obj) for obj, _ in results], "-Xlinker", "--exclude-libs=ALL", "-ldl"]
    res = subprocess.run(cmd, capture_output=True, text=True)
    if res.returncode != 0:
        raise RuntimeError(f"link failed:\n{res.stdout}\n{res.stderr}")
    return LIB_PATH


if __name__ == "__main__":
    path = build(force="--force" in sys.argv, verbose="-v" in sys.argv)
    print(path)
