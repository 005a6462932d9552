"""Build libbi_b200.so (the C-ABI kernel library) in-tree with nvcc for sm_100a, and beside it the CPython face of its hot
entry points (csrc/calls.c) for the interpreter that runs this, named with its ABI tag.

    python -m mlx_batch_invariant_b200.build          # rebuild if sources changed
    python -m mlx_batch_invariant_b200.build --force

nvcc cross-compiles without a GPU. The .so lands next to this file so it travels
with the source tree; nothing is written outside the package directory.
"""

from __future__ import annotations

import hashlib
import os
import shutil
import subprocess
import sys
import sysconfig
from concurrent.futures import ThreadPoolExecutor
from pathlib import Path

PKG = Path(__file__).resolve().parent
CSRC = PKG / "csrc"
OUT = PKG / "libbi_b200.so"
CALLS = PKG / ("_calls" + sysconfig.get_config_var("EXT_SUFFIX"))     # another Python version looks for another name
OBJ = PKG / "build"
SOURCES = ["abi.cu", "rmsnorm.cu", "attention.cu", "attn_prefill.cu", "attn_decode_static.cu", "matmul_simt.cu", "matmul_tc.cu", "matmul_pair.cu", "dequant.cu", "matmul.cu", "glue.cu", "peer.cu"]

# No fast-math anywhere: IEEE divide / sqrt, denormals kept, and fma contraction off so
# the only fused operations are the ones the sources spell out.
NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17", "-lineinfo",
    "-Xcompiler", "-fPIC", "--fmad=false", "--prec-div=true", "--prec-sqrt=true", "--ftz=false",
]


def _nvcc() -> str:
    for cand in (os.environ.get("NVCC"), shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if cand and os.path.exists(cand):
            return cand
    raise RuntimeError("nvcc not found (set NVCC=/path/to/nvcc)")


def _sources() -> list[Path]:
    return [CSRC / s for s in SOURCES if (CSRC / s).exists()]


def _fingerprint(sources: list[Path], *flags: str) -> str:
    h = hashlib.sha256()
    for p in sorted(sources + [PKG.parent / "include" / "bi_abi.h"]):
        h.update(p.name.encode())
        h.update(p.read_bytes())
    h.update(" ".join(flags).encode())
    return h.hexdigest()


def _is_fresh(out: Path, stamp: Path, fp: str) -> bool:
    return out.exists() and stamp.exists() and stamp.read_text() == fp


def build_calls(force: bool = False) -> Path:
    """The CPython module, by nvcc's host compiler (what links the library also compiles this); rebuilt on its own. Without
    Python's headers there is none, and _lib.py calls the library through ctypes."""
    src = CSRC / "calls.c"
    flags = ["-shared", "-cudart", "none", "-O2", "-Xcompiler", "-fPIC,-Wall", "-I", sysconfig.get_paths()["include"]]
    stamp, fp = OBJ / (CALLS.name + ".txt"), _fingerprint([src], *flags, sys.version)
    (PKG / "_calls.so").unlink(missing_ok=True)          # without a tag any Python would import it
    if force or not _is_fresh(CALLS, stamp, fp):
        if not (Path(flags[-1]) / "Python.h").exists():
            sys.stderr.write(f"no Python.h in {flags[-1]}: {CALLS.name} is not built\n")
            return CALLS
        OBJ.mkdir(exist_ok=True)
        r = subprocess.run([_nvcc(), *flags, "-o", str(CALLS), str(src), "-ldl"], capture_output=True, text=True)
        if r.returncode != 0:
            raise RuntimeError(f"nvcc failed for {src.name}:\n{r.stdout}\n{r.stderr}")
        stamp.write_text(fp)
    return CALLS


def build(force: bool = False, verbose: bool = False) -> Path:
    build_calls(force)
    stamp = OBJ / "fingerprint.txt"
    fp = _fingerprint(list(CSRC.glob("*.cu")) + list(CSRC.glob("*.cuh")), *NVCC_FLAGS)
    if not force and _is_fresh(OUT, stamp, fp):
        return OUT
    OBJ.mkdir(exist_ok=True)
    nvcc = _nvcc()

    def compile_one(src: Path) -> Path:
        obj = OBJ / (src.stem + ".o")
        cmd = [nvcc, *NVCC_FLAGS, "-c", str(src), "-o", str(obj)]
        if verbose:
            cmd.insert(1, "-Xptxas=-v")
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode != 0:
            raise RuntimeError(f"nvcc failed for {src.name}:\n{r.stdout}\n{r.stderr}")
        if verbose:
            sys.stderr.write(r.stderr)
        return obj

    with ThreadPoolExecutor(max_workers=min(8, os.cpu_count() or 1)) as ex:
        objs = list(ex.map(compile_one, _sources()))
    r = subprocess.run([nvcc, "-shared", "-o", str(OUT), *map(str, objs)], capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError(f"link failed:\n{r.stdout}\n{r.stderr}")
    stamp.write_text(fp)
    return OUT


if __name__ == "__main__":
    path = build(force="--force" in sys.argv, verbose="-v" in sys.argv)
    print(path)
