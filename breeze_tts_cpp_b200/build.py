"""Builds libb200q.so (the CUDA kernels + C++ host layer + C ABI) in-tree for sm_100a, and beside it the
CPython binding _native.so that ops.py calls per operation.

Run as `python -m breeze_tts_cpp_b200.build`. Objects are rebuilt only when a source or header
is newer; the producers are compiled with --fmad=false like the reference's own producers
(reference: CMakeLists.txt:94-105), the GEMM with default contraction.
"""
from __future__ import annotations

import os
import shutil
import subprocess
import sys
import sysconfig
from concurrent.futures import ThreadPoolExecutor
from pathlib import Path

HERE = Path(__file__).resolve().parent
CSRC = HERE / "csrc"
INCLUDE = HERE.parent / "include"
OBJ = HERE / "build"
LIB = HERE / "libb200q.so"
BINDING_SOURCE = CSRC / "bindings" / "python.cpp"
BINDING = HERE / "_native.so"  # the CPython side of ops.py, linked against libb200q.so beside it
ARCH = ["-gencode", "arch=compute_100a,code=sm_100a"]

# (source, extra flags)
SOURCES = [
    ("kernels/row_quantize.cu", ["--fmad=false"]),
    ("kernels/quant_norm.cu", ["--fmad=false"]),
    ("kernels/quant_gated.cu", ["--fmad=false"]),
    ("kernels/quant_linear.cu", []),
    ("kernels/quant_linear_dense.cu", []),
    ("kernels/quant_linear_static.cu", []),
    ("ops/quantized_gemm.cpp", []),
    ("ops/quantization_policy.cpp", []),
    ("ops/context.cpp", []),
    ("ops/ops.cpp", []),
    ("ops/sequence.cpp", []),
    ("kernels/sequence_pointwise.cu", ["--fmad=false"]),
    ("kernels/sequence_norm.cu", ["--fmad=false"]),
    ("layers/linear.cpp", []),
    ("c_api.cpp", []),
]


def _nvcc() -> str:
    found = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(found):
        raise RuntimeError("nvcc not found; the CUDA toolkit is required to build libb200q.so")
    return found


def _newest_header() -> float:
    stamps = [p.stat().st_mtime for p in list(CSRC.rglob("*.h")) + list(CSRC.rglob("*.cuh")) + list(INCLUDE.glob("*.h"))]
    return max(stamps) if stamps else 0.0


def _compile(nvcc: str, source: str, flags: list[str], header_stamp: float, verbose: bool) -> Path:
    src = CSRC / source
    obj = OBJ / (source.replace("/", "_") + ".o")
    if obj.exists() and obj.stat().st_mtime >= max(src.stat().st_mtime, header_stamp):
        return obj
    cmd = [nvcc, "-std=c++17", "-O3", *ARCH, "-lineinfo", "-Xcompiler", "-fPIC", f"-I{CSRC}", f"-I{INCLUDE}",
           *flags, *os.environ.get("B200Q_NVCC_FLAGS", "").split(), "-c", str(src), "-o", str(obj)]
    if verbose:
        print(" ".join(cmd), flush=True)
    done = subprocess.run(cmd, capture_output=True, text=True)
    if done.returncode:
        raise RuntimeError(f"nvcc failed on {source}:\n{done.stdout}\n{done.stderr}")
    return obj


def build(verbose: bool = False, force: bool = False) -> Path:
    nvcc = _nvcc()
    OBJ.mkdir(exist_ok=True)
    sources = [(s, f) for s, f in SOURCES if (CSRC / s).exists()]
    if force:
        for o in OBJ.glob("*.o"):
            o.unlink()
    stamp = _newest_header()
    with ThreadPoolExecutor(max_workers=min(8, len(sources))) as pool:
        objects = list(pool.map(lambda sf: _compile(nvcc, sf[0], sf[1], stamp, verbose), sources))
    if not LIB.exists() or any(LIB.stat().st_mtime < o.stat().st_mtime for o in objects):
        cmd = [nvcc, "-shared", *ARCH, "-o", str(LIB), *map(str, objects), "-lcudart"]
        if verbose:
            print(" ".join(cmd), flush=True)
        done = subprocess.run(cmd, capture_output=True, text=True)
        if done.returncode:
            raise RuntimeError(f"link failed:\n{done.stdout}\n{done.stderr}")
    _build_binding(verbose, force)
    return LIB


def _build_binding(verbose: bool, force: bool = False) -> None:
    """The binding calls the C ABI only, so of this library's files its own source and the ABI's header matter. It is compiled
    against one Python and one torch: the command and both versions are kept beside the objects, and others rebuild it."""
    import torch
    from torch.utils import cpp_extension
    torch_lib = Path(torch.__file__).parent / "lib"
    cmd = ["g++", "-std=c++17", "-O2", "-fPIC", "-shared", f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
           f"-I{INCLUDE}", f"-I{sysconfig.get_paths()['include']}", *(f"-isystem{p}" for p in cpp_extension.include_paths()),
           str(BINDING_SOURCE), "-o", str(BINDING), f"-L{HERE}", "-l:libb200q.so", "-Wl,-rpath,$ORIGIN",
           f"-L{torch_lib}", "-ltorch_python", "-ltorch_cpu", "-lc10"]
    key = "\n".join([torch.__version__, sysconfig.get_config_var("SOABI") or "", *cmd])
    made_with = OBJ / "binding.key"
    stamp = max(p.stat().st_mtime for p in (BINDING_SOURCE, INCLUDE / "b200q.h"))
    if not force and BINDING.exists() and BINDING.stat().st_mtime >= stamp and made_with.exists() and made_with.read_text() == key:
        return
    if verbose:
        print(" ".join(cmd), flush=True)
    done = subprocess.run(cmd, capture_output=True, text=True)
    if done.returncode:
        raise RuntimeError(f"building the Python binding failed:\n{done.stdout}\n{done.stderr}")
    made_with.write_text(key)


if __name__ == "__main__":
    print(build(verbose=True, force="--force" in sys.argv))
