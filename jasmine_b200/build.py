"""Build recipe of libjasmine_b200.so (CUDA kernels + C ABI) for sm_100a.

Each .cu file under csrc/ is compiled to an object with nvcc (in parallel) and
the objects are linked into jasmine_b200/libjasmine_b200.so.  The CUDA runtime
is linked statically and the driver API is reached through
cudaGetDriverEntryPoint, so the library loads on a machine without a GPU
driver (compute calls then return JSM_CUDA).

The frequent calls of the Python plumbing are a small extension module beside it (csrc/py_calls.cpp -> jasmine_b200/_native.so, g++
against the headers of the installed torch); where torch is not installed, or the module cannot be built, it is left out (with a word on
stderr), and the plumbing goes through ctypes.

Run as `python -m jasmine_b200.build [--force] [--verbose]`.
"""
from __future__ import annotations

import concurrent.futures as cf
import hashlib
import importlib.util
import os
import re
import shutil
import subprocess
import sys
import sysconfig
from pathlib import Path

PKG = Path(__file__).resolve().parent
CSRC = PKG / "csrc"
OBJ = PKG / "build"
LIB = PKG / "libjasmine_b200.so"
CALLS = PKG / "_native.so"

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a",
    "-std=c++20", "-O3", "-lineinfo",
    "-Xcompiler", "-fPIC,-fvisibility=hidden",
    "--expt-relaxed-constexpr",
    "-Xptxas", "-v",
]


def _nvcc() -> str:
    for cand in (os.environ.get("NVCC"), "/usr/local/cuda/bin/nvcc", "nvcc"):
        if cand and (os.path.sep not in cand or os.path.exists(cand)):
            return cand
    raise RuntimeError("nvcc not found")


def _stamp(src: Path) -> str:
    h = hashlib.sha256()
    h.update(" ".join(NVCC_FLAGS).encode())
    h.update(src.read_bytes())
    for hdr in sorted(list(CSRC.glob("*.cuh")) + list(CSRC.glob("*.h")) + [PKG.parent / "include" / "jasmine_b200.h"]):
        h.update(hdr.read_bytes())
    return h.hexdigest()


def _compile(src: Path, force: bool, verbose: bool) -> Path:
    obj = OBJ / (src.stem + ".o")
    stamp_file = OBJ / (src.stem + ".stamp")
    stamp = _stamp(src)
    if not force and obj.exists() and stamp_file.exists() and stamp_file.read_text() == stamp:
        return obj
    cmd = [_nvcc(), *NVCC_FLAGS, "-c", str(src), "-o", str(obj)]
    res = subprocess.run(cmd, capture_output=True, text=True)
    (OBJ / (src.stem + ".ptxas.log")).write_text(res.stderr)
    if res.returncode != 0:
        raise RuntimeError(f"nvcc failed for {src.name}:\n{res.stderr[-6000:]}")
    if verbose:
        print(res.stderr)
    stamp_file.write_text(stamp)
    return obj


def _torch_id(torch: Path) -> str:
    """What a torch says it is, `<version> <revision>`, without importing it."""
    text = (torch / "version.py").read_text()
    return " ".join(re.search(rf"^{name}\b[^=\n]*=\s*['\"]([^'\"]*)['\"]", text, re.M)[1] for name in ("__version__", "git_version"))


def _build_calls(force: bool) -> None:
    spec = importlib.util.find_spec("torch")
    if spec is None or not spec.submodule_search_locations:
        return
    torch = Path(spec.submodule_search_locations[0])
    nvcc = shutil.which(_nvcc())
    cuda = Path(nvcc).resolve().parents[1] if nvcc else Path("/usr/local/cuda")
    src, built_for = CSRC / "py_calls.cpp", _torch_id(torch)
    cmd = [os.environ.get("CXX", "g++"), "-std=c++17", "-O2", "-fPIC", "-shared", "-fvisibility=hidden", f'-DJSM_TORCH="{built_for}"',
           "-I" + sysconfig.get_paths()["include"], f"-I{torch}/include", f"-I{torch}/include/torch/csrc/api/include", f"-I{cuda}/include", str(src), "-o", str(CALLS),
           f"-L{torch}/lib", "-ltorch_python", "-ltorch", "-ltorch_cpu", "-lc10", "-lc10_cuda"]
    stamp = hashlib.sha256(" ".join([*cmd, sys.version]).encode() + src.read_bytes() + (PKG.parent / "include" / "jasmine_b200.h").read_bytes()).hexdigest()
    stamp_file = OBJ / "py_calls.stamp"
    if not force and CALLS.exists() and stamp_file.exists() and stamp_file.read_text() == stamp:
        return
    CALLS.unlink(missing_ok=True)  # (nothing older than its sources stays behind a failure)
    res = subprocess.run(cmd, capture_output=True, text=True)
    if res.returncode != 0:
        CALLS.unlink(missing_ok=True)
        raise RuntimeError(f"{cmd[0]} failed for {src.name}:\n{res.stderr[-6000:]}")
    stamp_file.write_text(stamp)


def build(force: bool = False, verbose: bool = False) -> Path:
    OBJ.mkdir(exist_ok=True)
    sources = sorted(CSRC.glob("*.cu"))
    with cf.ThreadPoolExecutor(max_workers=min(8, len(sources))) as ex:
        calls = ex.submit(_build_calls, force)
        objs = list(ex.map(lambda s: _compile(s, force, verbose), sources))
    newest = max(o.stat().st_mtime for o in objs)
    if force or not LIB.exists() or LIB.stat().st_mtime < newest:
        cmd = [_nvcc(), "-shared", "-o", str(LIB), *map(str, objs), "-cudart", "static",
               "-Xlinker", "--no-undefined", "-lpthread", "-ldl", "-lrt"]
        res = subprocess.run(cmd, capture_output=True, text=True)
        if res.returncode != 0:
            raise RuntimeError(f"link failed:\n{res.stderr[-4000:]}")
    try:
        calls.result()
    except Exception as e:  # the library does without it
        print(f"jasmine_b200: {CALLS.name} was not built, the Python plumbing goes through ctypes: {e}", file=sys.stderr)
    return LIB


if __name__ == "__main__":
    lib = build(force="--force" in sys.argv, verbose="--verbose" in sys.argv)
    print(lib)
