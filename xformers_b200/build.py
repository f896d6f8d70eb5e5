"""Build recipe of libxfb200.so (the C-ABI library holding every CUDA kernel)
and of the extension module ``_front`` (the operators' host front).

``python -m xformers_b200.build`` compiles ``csrc/*.cu`` for sm_100a with nvcc
and links them into ``csrc/libxfb200.so`` next to the sources, and
``csrc/front.cpp`` against the torch headers into ``_front.so``, so that both are
found in-tree.  nvcc cross-compiles without a GPU.
"""

from __future__ import annotations

import concurrent.futures
import hashlib
import os
import shutil
import subprocess
import sys
import sysconfig
from pathlib import Path

CSRC = Path(__file__).resolve().parent / "csrc"
LIB = CSRC / "libxfb200.so"
FRONT = CSRC.parent / "_front.so"
SOURCES = [
    "runtime.cu",
    "merge.cu",
    "decode_splitk.cu",
    "prefill_generic.cu",
    "prefill_sm100_host.cu",
    "prefill_sm100_m256.cu",
    "prefill_sm100_persist.cu",
    "prefill_api.cu",
    "rope_padded.cu",
]
HEADERS = ["internal.h", "ptx.cuh", "prefill_sm100.h", "../../include/xfb200.h"]
NVCC_FLAGS = [
    "-gencode",
    "arch=compute_100a,code=sm_100a",
    "-lineinfo",
    "-O3",
    "-std=c++17",
    "--use_fast_math",
    "-Xcompiler",
    "-fPIC",
    "-Xcompiler",
    "-fvisibility=hidden",
    # a function that can fall off its end without a return value is an error, not a warning
    "-Xcompiler",
    "-Werror=return-type",
    "-Werror",
    "cross-execution-space-call",
]


def _nvcc() -> str:
    exe = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(exe):
        raise RuntimeError("nvcc not found: libxfb200.so cannot be built")
    return exe


def _stamp() -> str:
    h = hashlib.sha256()
    for name in SOURCES + HEADERS:
        h.update((CSRC / name).read_bytes())
    h.update(" ".join(NVCC_FLAGS).encode())
    return h.hexdigest()


def build_front(force: bool = False) -> Path:
    """The extension module: host code only, it reaches the kernels through the addresses it is given."""
    import torch

    root = Path(torch.__file__).resolve().parent
    cuda = Path(_nvcc()).resolve().parent.parent
    cmd = ["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-fvisibility=hidden", "-DTORCH_EXTENSION_NAME=_front", "-DTORCH_API_INCLUDE_EXTENSION_H",
           f"-D_GLIBCXX_USE_CXX11_ABI={int(torch.compiled_with_cxx11_abi())}", f"-I{root}/include", f"-I{root}/include/torch/csrc/api/include",
           f"-I{sysconfig.get_paths()['include']}", f"-I{cuda}/include", str(CSRC / "front.cpp"), "-o", str(FRONT), f"-L{root}/lib", "-lc10", "-lc10_cuda",
           "-ltorch_cpu", "-ltorch_cuda", "-ltorch", "-ltorch_python", f"-Wl,-rpath,{root}/lib"]
    h = hashlib.sha256()
    for name in ("front.cpp", "../../include/xfb200.h"):
        h.update((CSRC / name).read_bytes())
    stamp = h.hexdigest() + torch.__version__ + sys.version + " ".join(cmd)
    stamp_file = CSRC / "build" / "front_stamp"
    if not force and FRONT.exists() and stamp_file.exists() and stamp_file.read_text() == stamp:
        return FRONT
    stamp_file.parent.mkdir(parents=True, exist_ok=True)
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError(f"g++ failed on front.cpp:\n{r.stdout}\n{r.stderr}")
    stamp_file.write_text(stamp)
    return FRONT


def build(force: bool = False, verbose: bool = False, extra_flags=(), out: Path = LIB) -> Path:
    """``extra_flags`` / ``out`` build an experimental variant beside the
    default library (selected at run time with XFB200_LIBRARY)."""
    with concurrent.futures.ThreadPoolExecutor(max_workers=1) as ex:
        front = ex.submit(build_front, force)
        lib = _build_lib(force, verbose, extra_flags, out)
        front.result()
    return lib


def _build_lib(force: bool, verbose: bool, extra_flags, out: Path) -> Path:
    variant = bool(extra_flags) or Path(out) != LIB
    objdir = CSRC / "build" / (hashlib.sha256(" ".join(extra_flags).encode()).hexdigest()[:8] if variant else "")
    stamp_file = objdir / "stamp"
    stamp = _stamp() + " ".join(extra_flags)
    if not force and Path(out).exists() and stamp_file.exists() and stamp_file.read_text() == stamp:
        return Path(out)
    objdir.mkdir(parents=True, exist_ok=True)
    nvcc = _nvcc()

    def compile_one(src: str) -> Path:
        obj = objdir / (Path(src).stem + ".o")
        cmd = [nvcc, *NVCC_FLAGS, *extra_flags, "-c", str(CSRC / src), "-o", str(obj)]
        if verbose:
            cmd.insert(1, "-Xptxas=-v")
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode != 0:
            raise RuntimeError(f"nvcc failed on {src}:\n{r.stdout}\n{r.stderr}")
        if verbose:
            sys.stderr.write(r.stderr)
        return obj

    with concurrent.futures.ThreadPoolExecutor(max_workers=min(8, len(SOURCES))) as ex:
        objs = list(ex.map(compile_one, SOURCES))
    cmd = [nvcc, "-shared", "-o", str(out), *map(str, objs)]
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError(f"link failed:\n{r.stdout}\n{r.stderr}")
    stamp_file.write_text(stamp)
    return Path(out)


if __name__ == "__main__":
    defs = [a for a in sys.argv[1:] if a.startswith("-D")]
    outs = [a.split("=", 1)[1] for a in sys.argv[1:] if a.startswith("--out=")]
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv, extra_flags=tuple(defs), out=Path(outs[0]) if outs else LIB))
