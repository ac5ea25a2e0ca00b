"""In-tree build of the CUDA library (sm_103a).

`build_library()` compiles opensayal_gb300/csrc into
opensayal_gb300/lib/libopensayal_gb300.so with nvcc, for GB300 only
(`-gencode arch=compute_103a,code=sm_103a`) and with `--use_fast_math`, the
reference's own Release flag (CMakeLists.txt:21), so that FP32 divisions and
square roots round the way the reference's kernels do.
"""
from __future__ import annotations

import os
import shutil
import subprocess
import tempfile
from concurrent.futures import ThreadPoolExecutor
from pathlib import Path

PKG = Path(__file__).resolve().parent
ROOT = PKG.parent
CSRC = PKG / "csrc"
LIB_DIR = PKG / "lib"
LIB_PATH = LIB_DIR / "libopensayal_gb300.so"
HEADER = ROOT / "include" / "opensayal_gb300.h"

ARCH_FLAGS = ["-gencode", "arch=compute_103a,code=sm_103a"]
NVCC_FLAGS = [
    "-std=c++17", "-O3", "--use_fast_math", "-lineinfo",
    "-Xcompiler", "-fPIC", "-diag-suppress", "177",
]

# Translation units, compiled side by side: (source, defines). The tile kernels
# take one unit per strip height.
TILE_ROWS = {"project": (10, 8, 6, 4, 2), "diffuse": (12, 8, 6, 4, 2)}
UNITS = [("os_fluid.cu", ()), ("os_tile_batch.cu", ())]
UNITS += [(f"os_tile_{phase}.cu", (f"OS_TILE_ROWS={rows}",))
          for phase, heights in TILE_ROWS.items() for rows in heights]


def _nvcc() -> str:
    cuda_home = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    cand = Path(cuda_home) / "bin" / "nvcc"
    if cand.exists():
        return str(cand)
    found = shutil.which("nvcc")
    if not found:
        raise RuntimeError("nvcc not found: the GB300 library cannot be built")
    return found


def _sources() -> list[Path]:
    return sorted(CSRC.glob("*.cu")) + sorted(CSRC.glob("*.cuh")) + [HEADER]


def _stale(target: Path, deps: list[Path]) -> bool:
    if not target.exists():
        return True
    t = target.stat().st_mtime
    return any(d.stat().st_mtime > t for d in deps)


def _run(cmd: list[str], verbose: bool) -> None:
    res = subprocess.run(cmd, capture_output=True, text=True)
    if res.returncode != 0:
        raise RuntimeError(f"nvcc failed ({' '.join(cmd)}):\n{res.stdout}\n{res.stderr}")
    if verbose:
        print(res.stderr)


def build_library(force: bool = False, verbose: bool = False) -> Path:
    """Compile the library if any source is newer than the built .so."""
    if not force and not _stale(LIB_PATH, _sources()):
        return LIB_PATH
    LIB_DIR.mkdir(parents=True, exist_ok=True)
    tmp = LIB_PATH.with_suffix(".so.tmp")
    with tempfile.TemporaryDirectory(dir=LIB_DIR) as work:
        def compile_unit(index: int) -> str:
            source, defines = UNITS[index]
            obj = str(Path(work) / f"{index}.o")
            cmd = [_nvcc(), *NVCC_FLAGS, *ARCH_FLAGS, *(f"-D{d}" for d in defines),
                   *(["-Xptxas=-v"] if verbose else []), "-c", "-o", obj, str(CSRC / source)]
            _run(cmd, verbose)
            return obj

        with ThreadPoolExecutor(max_workers=os.cpu_count() or 1) as pool:
            objects = list(pool.map(compile_unit, range(len(UNITS))))
        _run([_nvcc(), *ARCH_FLAGS, "-shared", "-o", str(tmp), *objects], verbose)
    os.replace(tmp, LIB_PATH)
    return LIB_PATH


if __name__ == "__main__":
    print(build_library(force=True, verbose=True))
