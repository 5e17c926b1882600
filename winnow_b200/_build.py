"""Build recipe: libwinnow_tq.so (the kernels, nvcc, sm_100a only) and _host.so
(the native host side of the Python operators, g++ against torch's headers),
both in-tree next to this file."""
from __future__ import annotations

import os
import shutil
import subprocess
import sysconfig
import tempfile
from concurrent.futures import ThreadPoolExecutor
from pathlib import Path

PKG = Path(__file__).resolve().parent
CSRC = PKG / "csrc"
LIB = PKG / "libwinnow_tq.so"
HOST = PKG / "_host.so"
SOURCES = ["wtq_pack.cu", "wtq_append.cu", "wtq_quant_mma.cu", "wtq_decode.cu", "wtq_decode_mma.cu", "wtq_decode_fused.cu",
           "wtq_api.cu", "wtq_dequant.cu", "wtq_dequant_umma.cu", "wtq_prefill.cu", "wtq_rows_mma.cu",
           "wtq_decode_static.cu", "wtq_dense.cu"]
NVCC_FLAGS = ["-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
              "-Xcompiler", "-fPIC"]


def _nvcc() -> str | None:
    return shutil.which("nvcc") or (
        "/usr/local/cuda/bin/nvcc" if os.path.exists("/usr/local/cuda/bin/nvcc") else None)


def sources() -> list[Path]:
    return [CSRC / s for s in SOURCES]


def up_to_date() -> bool:
    if not LIB.exists() or not HOST.exists():
        return False
    built = min(LIB.stat().st_mtime, HOST.stat().st_mtime)
    deps = list(CSRC.glob("*.cu")) + list(CSRC.glob("*.cuh")) + list(CSRC.glob("*.cpp")) \
        + [PKG.parent / "include" / "winnow_tq.h"]
    return all(d.stat().st_mtime <= built for d in deps)


def _run(cmd: list[str]) -> str:
    proc = subprocess.run(cmd, capture_output=True, text=True)
    if proc.returncode != 0:
        raise RuntimeError(f"{cmd[0]} failed:\n{proc.stdout}\n{proc.stderr}")
    return proc.stderr


def host_command(out: Path = HOST) -> list[str]:
    from torch.utils import cpp_extension
    includes = [f"-I{p}" for p in cpp_extension.include_paths(device_type="cuda")]
    libs = [p for d in cpp_extension.library_paths(device_type="cuda") for p in (f"-L{d}", f"-Wl,-rpath,{d}")]
    return ["g++", "-O2", "-std=c++17", "-shared", "-fPIC", *includes,
            f"-I{sysconfig.get_paths()['include']}", "-o", str(out), str(CSRC / "host.cpp"), str(LIB),
            "-Wl,-rpath,$ORIGIN", *libs, "-lc10", "-lc10_cuda", "-ltorch", "-ltorch_cpu", "-ltorch_cuda",
            "-ltorch_python"]


def build(force: bool = False, verbose: bool = False) -> Path:
    """Compile every kernel into one shared library next to this file (sources in
    parallel, then one link), then the host module against it."""
    if not force and up_to_date():
        return LIB
    nvcc = _nvcc()
    if nvcc is None:
        raise RuntimeError("nvcc not found: cannot build libwinnow_tq.so")
    flags = [*NVCC_FLAGS, *(["-Xptxas", "-v"] if verbose else [])]
    with tempfile.TemporaryDirectory() as tmp, ThreadPoolExecutor(os.cpu_count() or 4) as pool:
        objects = [str(Path(tmp) / (s + ".o")) for s in SOURCES]
        logs = list(pool.map(lambda so: _run([nvcc, *flags, "-c", "-o", so[1], str(so[0])]),
                             zip(sources(), objects)))
        if verbose:
            print("".join(logs))
        _run([nvcc, *NVCC_FLAGS, "-shared", "-Xlinker", f"-soname={LIB.name}", "-o", str(LIB), *objects])
    _run(host_command())
    return LIB
