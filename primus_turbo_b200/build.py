"""Build recipe for the in-tree libraries (sm_100a only).

``python -m primus_turbo_b200.build`` compiles ``csrc/*.cu`` with nvcc into
``primus_turbo_b200/_C/libptb_b200.so`` (the C ABI, no torch in it) and ``csrc/torch_ops.cpp`` with the host
compiler into ``_C/ptb_torch.so`` (the native host path of the torch ops, linked against the former).  nvcc
cross-compiles, so no GPU is needed to build.
"""

from __future__ import annotations

import os
import shutil
import subprocess
import sys
import sysconfig
from pathlib import Path

PKG_DIR = Path(__file__).resolve().parent
REPO_DIR = PKG_DIR.parent
CSRC = PKG_DIR / "csrc"
OUT_DIR = PKG_DIR / "_C"
LIB_PATH = OUT_DIR / "libptb_b200.so"
EXT_PATH = OUT_DIR / "ptb_torch.so"
EXT_SOURCE = CSRC / "torch_ops.cpp"

SOURCES = ["ptb_quant.cu", "ptb_gemm.cu", "ptb_exchange.cu", "ptb_activation.cu", "ptb_mxfp8.cu"]
NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a",
    "-lineinfo", "-O3", "-std=c++17",
    "-Xcompiler", "-fPIC",
    "-Xcompiler", "-fvisibility=hidden",
]


def _nvcc() -> str:
    for cand in (os.environ.get("NVCC"), shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if cand and os.path.exists(cand):
            return cand
    raise RuntimeError("nvcc not found; set NVCC or put it on PATH")


def _newer(deps, target: Path) -> bool:
    return not target.exists() or any(d.stat().st_mtime > target.stat().st_mtime for d in deps)


def needs_build() -> bool:
    header = REPO_DIR / "include" / "ptb.h"
    return _newer([CSRC / s for s in SOURCES] + list(CSRC.glob("*.cuh")) + [header], LIB_PATH) or _newer(
        [EXT_SOURCE, header], EXT_PATH
    )


def _extension_command():
    import torch
    from torch.utils.cpp_extension import include_paths

    torch_lib = Path(torch.__file__).parent / "lib"
    cuda = Path(_nvcc()).resolve().parent.parent
    includes = [str(REPO_DIR / "include"), *include_paths(), str(cuda / "include"), sysconfig.get_paths()["include"]]
    return [
        os.environ.get("CXX", "g++"), "-O2", "-std=c++17", "-fPIC", "-shared", "-fvisibility=hidden",
        f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}", "-DTORCH_EXTENSION_NAME=ptb_torch",
        *(f"-I{i}" for i in includes), str(EXT_SOURCE), "-o", str(EXT_PATH), f"-L{OUT_DIR}", "-lptb_b200", f"-L{torch_lib}",
        "-ltorch", "-ltorch_cpu", "-ltorch_cuda", "-lc10", "-lc10_cuda", "-ltorch_python", "-Wl,-rpath,$ORIGIN",
    ]


def _run(cmd, what: str) -> None:
    r = subprocess.run(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)
    if r.returncode != 0:
        raise RuntimeError(f"{what} failed: {' '.join(cmd)}\n{r.stdout}")


def build(force: bool = False, verbose: bool = False) -> Path:
    if not force and not needs_build():
        return LIB_PATH
    OUT_DIR.mkdir(exist_ok=True)
    nvcc = _nvcc()
    header = REPO_DIR / "include" / "ptb.h"
    shared = list(CSRC.glob("*.cuh")) + [header]
    objs = []
    procs = []
    for src in SOURCES:
        obj = OUT_DIR / (Path(src).stem + ".o")
        objs.append(str(obj))
        if not force and not _newer([CSRC / src, *shared], obj):
            continue
        cmd = [nvcc, *NVCC_FLAGS, f"-I{REPO_DIR / 'include'}", f"-I{CSRC}", "-c", str(CSRC / src), "-o", str(obj)]
        if verbose:
            cmd.insert(1, "-Xptxas=-v")
        procs.append((cmd, subprocess.Popen(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)))
    for cmd, p in procs:
        out, _ = p.communicate()
        if verbose and out:
            print(out)
        if p.returncode != 0:
            raise RuntimeError(f"nvcc failed: {' '.join(cmd)}\n{out}")
    soname = ["-Xlinker", "-soname", "-Xlinker", LIB_PATH.name]
    _run([nvcc, "-shared", "-gencode", "arch=compute_100a,code=sm_100a", *soname, "-o", str(LIB_PATH), *objs], "link")
    if force or _newer([EXT_SOURCE, header], EXT_PATH):
        _run(_extension_command(), "host compiler")
    return LIB_PATH


if __name__ == "__main__":
    path = build(force="--force" in sys.argv, verbose="-v" in sys.argv)
    print(path)
