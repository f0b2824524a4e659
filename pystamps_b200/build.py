"""Build libps2cuda.so in-tree with nvcc for sm_100a (no GPU needed)."""
from __future__ import annotations

import os
import shutil
import subprocess
import tempfile
from concurrent.futures import ThreadPoolExecutor
from pathlib import Path

HERE = Path(__file__).resolve().parent
CSRC = HERE / "csrc"
SOURCES = [CSRC / "ps2_kernels.cu", CSRC / "ps2_api.cu", CSRC / "clap_f32.cu", CSRC / "topofit_f32.cu", CSRC / "v5_uniform.cu"]
HEADERS = [CSRC / "ps2_kernels.cuh", CSRC / "ps2_device.cuh", CSRC / "v5_uniform.cuh", CSRC / "clap_f32.cuh", CSRC / "phase_math.cuh", CSRC / "interp10_taps.h", CSRC / "trial_interp_taps.h", CSRC / "sincos_poly.h", CSRC / "atan_poly.h",
           HERE.parent / "include" / "ps2cuda.h"]
TARGET = HERE / "libps2cuda.so"

NVCC_FLAGS = [
    "-O3", "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo",
    "-Xcompiler", "-fPIC", "-shared",
]


def nvcc() -> str:
    for cand in (os.environ.get("NVCC"), shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if cand and Path(cand).exists():
            return cand
    raise RuntimeError("nvcc not found")


def needs_build() -> bool:
    if not TARGET.exists():
        return True
    t = TARGET.stat().st_mtime
    return any(p.stat().st_mtime > t for p in SOURCES + HEADERS)


def build(force: bool = False, verbose: bool = False) -> Path:
    if not force and not needs_build():
        return TARGET
    flags = [f for f in NVCC_FLAGS if f != "-shared"] + (["-Xptxas=-v"] if verbose else [])
    with tempfile.TemporaryDirectory() as tmp:  # one object per source, compiled side by side
        objs = [str(Path(tmp) / (s.stem + ".o")) for s in SOURCES]
        with ThreadPoolExecutor(len(SOURCES)) as ex:
            list(ex.map(lambda so: subprocess.run([nvcc(), *flags, "-c", "-o", so[1], str(so[0])], check=True, cwd=str(HERE)),
                        zip(SOURCES, objs)))
        subprocess.run([nvcc(), *NVCC_FLAGS, "-o", str(TARGET), *objs], check=True, cwd=str(HERE))
    return TARGET


if __name__ == "__main__":
    build(force=True, verbose=True)
    print(TARGET)
