"""Builds liboops_ta_sm100.so in-tree with nvcc for sm_100a (no GPU needed), and the host layer _native.so with g++.

    python -m oops_b200.csrc.build [--force]

Both land in oops_b200/lib/.  The first is a plain C-ABI library (include/oops_ta.h); nothing in it links against Python
or PyTorch.  The second is the PyTorch extension over it (native.cpp).
"""

from __future__ import annotations

import importlib.util
import os
import subprocess
import sys
import sysconfig
from concurrent.futures import ThreadPoolExecutor
from pathlib import Path

CSRC = Path(__file__).resolve().parent
ROOT = CSRC.parent.parent
LIB_DIR = CSRC.parent / "lib"
LIB_PATH = LIB_DIR / "liboops_ta_sm100.so"
NATIVE_PATH = LIB_DIR / "_native.so"
SOURCES = ("ta_api.cu", "ta_generic.cu", "ta_f32.cu", "ta_mma.cu", "ta_gate.cu", "ta_mask.cu", "ta_bias.cu", "ta_layer_norm.cu", "ta_pair_update.cu", "ta_tensor_sm100.cu", "ta_tensor_bwd_sm100.cu", "ta_wide_sm100.cu", "ta_products_sm100.cu")
NVCC_FLAGS = (
    "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
    "-Xcompiler", "-fPIC", "--expt-relaxed-constexpr", "-Xptxas", "-v",
)


def _nvcc() -> str:
    cuda_home = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    candidate = Path(cuda_home) / "bin" / "nvcc"
    return str(candidate) if candidate.exists() else "nvcc"


# Kernels that keep tensor-memory loads in flight under arithmetic: a load writes its destination registers when the
# data arrives, so a spill (or copy) of such a register between issue and wait would save stale data.  ptxas must
# report no spill stores for them; the build fails otherwise.
NO_SPILL_KERNELS = ("ta_fwd_kernel", "ta_bwd_fused_kernel", "ta_bwd_dbias_kernel", "ta_wide_fwd_kernel", "ta_wide_bwd_kernel")


def _spilling_entries(ptxas_log: str, kernels) -> list:
    """Entry functions of `kernels` for which `ptxas -v` reports spill stores."""
    found, current = [], None
    for line in ptxas_log.splitlines():
        if "Compiling entry function" in line:
            current = line.split("'")[1] if "'" in line else line
        elif "bytes spill stores" in line and current is not None:
            stores = int(line.split("bytes stack frame,")[1].split("bytes spill stores")[0])
            if stores > 0 and any(k in current for k in kernels):
                found.append(f"{current}: {stores} bytes")
            current = None
    return found


def _stale(target: Path, deps) -> bool:
    if not target.exists():
        return True
    stamp = target.stat().st_mtime
    return any(Path(d).stat().st_mtime > stamp for d in deps)


def _native_commands(obj: Path) -> tuple:
    """Compile and link commands of the host layer; it finds the kernels' library beside itself."""
    torch_dir = Path(importlib.util.find_spec("torch").origin).parent
    cuda_home = Path(os.environ.get("CUDA_HOME", "/usr/local/cuda"))
    includes = (torch_dir / "include", torch_dir / "include/torch/csrc/api/include", sysconfig.get_paths()["include"], cuda_home / "include")
    compile_flags = ["-O2", "-std=c++17", "-fPIC", "-fvisibility=hidden", "-DTORCH_EXTENSION_NAME=_native", "-I", str(ROOT / "include")]
    compile_flags += [flag for path in includes for flag in ("-isystem", str(path))]
    libraries = ["-ltorch", "-ltorch_cpu", "-ltorch_cuda", "-ltorch_python", "-lc10", "-lc10_cuda"]
    link_flags = ["-L", str(LIB_DIR), "-L", str(torch_dir / "lib"), f"-l:{LIB_PATH.name}", *libraries, "-Wl,-rpath,$ORIGIN"]
    return (["g++", *compile_flags, "-c", str(CSRC / "native.cpp"), "-o", str(obj)],
            ["g++", "-shared", str(obj), "-o", str(NATIVE_PATH), *link_flags])


def _checked(cmd, what: str) -> None:
    done = subprocess.run(cmd, capture_output=True, text=True)
    if done.returncode != 0:
        raise RuntimeError(f"{what} failed:\n{done.stdout}\n{done.stderr}")


def build(force: bool = False, verbose: bool = False) -> Path:
    LIB_DIR.mkdir(exist_ok=True)
    obj_dir = LIB_DIR / "obj"
    obj_dir.mkdir(exist_ok=True)
    headers = [CSRC / "ta_internal.h", ROOT / "include" / "oops_ta.h", *CSRC.glob("*.cuh")]

    def compile_one(name: str):
        src = CSRC / name
        obj = obj_dir / (src.stem + ".o")
        if force or _stale(obj, [src, *headers]):
            cmd = [_nvcc(), *NVCC_FLAGS, "-I", str(ROOT / "include"), "-I", str(CSRC), "-c", str(src), "-o", str(obj)]
            done = subprocess.run(cmd, capture_output=True, text=True)
            log = obj_dir / (src.stem + ".ptxas.log")
            log.write_text(done.stdout + done.stderr)
            if done.returncode != 0:
                raise RuntimeError(f"nvcc failed for {name}:\n{done.stdout}\n{done.stderr}")
            spilled = _spilling_entries(done.stdout + done.stderr, NO_SPILL_KERNELS)
            if spilled:
                obj.unlink(missing_ok=True)
                raise RuntimeError(f"{name}: register spills in kernels that keep tensor-memory loads in flight: {spilled}")
            if verbose:
                print(done.stderr)
        return obj

    native_obj = obj_dir / "native.o"
    compile_native, link_native = _native_commands(native_obj)

    def compile_host():
        if force or _stale(native_obj, [CSRC / "native.cpp", ROOT / "include" / "oops_ta.h"]):
            _checked(compile_native, "g++ for native.cpp")

    with ThreadPoolExecutor(max_workers=len(SOURCES) + 1) as pool:
        host = pool.submit(compile_host)
        objects = list(pool.map(compile_one, SOURCES))
        host.result()
    if force or _stale(LIB_PATH, objects):
        _checked([_nvcc(), "-shared", "-o", str(LIB_PATH), *map(str, objects), "-lcudart"], "link")
    if force or _stale(NATIVE_PATH, [native_obj, LIB_PATH]):
        _checked(link_native, "link of the host layer")
    return LIB_PATH


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))
