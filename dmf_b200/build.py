"""Build the C-ABI shared library (dmf_b200/libdmf_attn.so) with nvcc for sm_100a, and the native host path of the Python
surface (dmf_b200/_dmf_torch.*.so, csrc/torch_host.cpp) with the C++ compiler.

Both are built in-tree so that they travel with the source snapshot.  The library has no Python or torch dependency; the
host module links it and torch, and has the Python and torch it was built for in its name: under others it is built anew.
``python -m dmf_b200.build`` builds them by hand.
"""

from __future__ import annotations

import fcntl
import os
import shutil
import subprocess
import sys
from pathlib import Path

PKG = Path(__file__).resolve().parent
CSRC = PKG / "csrc"
INCLUDE = PKG.parent / "include"
LIB = PKG / "libdmf_attn.so"

HOST_SOURCE = CSRC / "torch_host.cpp"

SOURCES = ["dmf_attn.cu", "attn_fwd_duo.cu", "dmf_adaln.cu", "dmf_step.cu"]
NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a",
    "-lineinfo", "-O3", "-std=c++17",
    "-Xcompiler", "-fPIC",
    "-Xcompiler", "-fvisibility=hidden",
    "-shared",
]


def find_nvcc() -> str | None:
    cand = os.environ.get("NVCC") or shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    return cand if cand and Path(cand).exists() else None


def host_module() -> Path:
    """The host module's path: it is compiled against torch's C++ internals and CPython's, so their versions name it."""
    import sysconfig

    import torch
    torch_id = f"torch{torch.__version__}-{(torch.version.git_version or '')[:8]}-cxx{int(torch.compiled_with_cxx11_abi())}"
    return PKG / f"_dmf_torch.{sysconfig.get_config_var('SOABI')}.{torch_id}.so"


def _older(target: Path, deps) -> bool:
    return not target.exists() or any(d.stat().st_mtime > target.stat().st_mtime for d in deps)


def _stale() -> bool:
    return _older(LIB, [*CSRC.glob("*.cu"), *CSRC.glob("*.cuh"), *CSRC.glob("*.h"), *INCLUDE.glob("*.h")])


def _host_stale() -> bool:
    return _older(host_module(), [HOST_SOURCE, *(CSRC / "compat").rglob("*.hpp"), *INCLUDE.glob("*.h")])


def build(force: bool = False, verbose: bool = False) -> Path:
    """Compile the library if it is missing or older than its sources.

    Several processes may get here at once (one rank per GPU under torchrun, spawned test workers): the stale
    check and the compile run under an exclusive lock on a sidecar file, so one process builds and the others
    wait and then find the library fresh; nvcc writes to a temporary name that is moved onto the library in
    one step, so nobody ever loads a half-written file.
    """
    if not force and not _stale():
        return LIB
    with open(PKG / ".build.lock", "w") as lock:
        fcntl.flock(lock, fcntl.LOCK_EX)
        try:
            if not force and not _stale():      # somebody else built it while this process waited
                return LIB
            nvcc = find_nvcc()
            if nvcc is None:
                raise RuntimeError("nvcc not found: cannot build dmf_b200/libdmf_attn.so")
            tmp = LIB.with_name(f".{LIB.name}.{os.getpid()}.tmp")
            cmd = [nvcc, *NVCC_FLAGS, f"-I{INCLUDE}", f"-I{CSRC}", "--threads", "0"]
            if verbose:
                cmd += ["-Xptxas", "-v"]
            cmd += ["-o", str(tmp), *[str(CSRC / s) for s in SOURCES]]
            res = subprocess.run(cmd, capture_output=True, text=True)
            if res.returncode != 0:
                tmp.unlink(missing_ok=True)
                raise RuntimeError(f"nvcc failed ({res.returncode}):\n{res.stdout}\n{res.stderr}")
            os.replace(tmp, LIB)
            if verbose:
                sys.stderr.write(res.stderr)
        finally:
            fcntl.flock(lock, fcntl.LOCK_UN)
    return LIB


def build_host(force: bool = False) -> Path:
    """Compile the native host path (torch_host.cpp) if it is missing or older than its sources; same locking as build()."""
    lib, target = build(), host_module()
    if not force and not _host_stale():
        return target
    import sysconfig

    import torch
    root = Path(torch.__file__).resolve().parent
    nvcc = find_nvcc()
    if nvcc is None:
        raise RuntimeError(f"no CUDA toolkit: cannot build {target.name}")
    with open(PKG / ".build.lock", "w") as lock:
        fcntl.flock(lock, fcntl.LOCK_EX)
        try:
            if not force and not _host_stale():
                return target
            tmp = target.with_name(f".{target.name}.{os.getpid()}.tmp")
            includes = [root / "include", root / "include" / "torch" / "csrc" / "api" / "include",
                        sysconfig.get_paths()["include"], Path(nvcc).resolve().parent.parent / "include", CSRC / "compat"]
            cmd = [os.environ.get("CXX", "g++"), "-O2", "-std=c++17", "-fPIC", "-shared", "-fvisibility=hidden",
                   "-DTORCH_EXTENSION_NAME=_dmf_torch", f"-D_GLIBCXX_USE_CXX11_ABI={int(torch.compiled_with_cxx11_abi())}",
                   *(f"-isystem{i}" for i in includes), f"-I{INCLUDE}", str(HOST_SOURCE), "-o", str(tmp), f"-L{root / 'lib'}",
                   "-ltorch", "-ltorch_cpu", "-ltorch_cuda", "-lc10", "-lc10_cuda", "-ltorch_python",
                   f"-L{lib.parent}", f"-l:{lib.name}", "-Wl,-rpath,$ORIGIN"]
            res = subprocess.run(cmd, capture_output=True, text=True)
            if res.returncode != 0:
                tmp.unlink(missing_ok=True)
                raise RuntimeError(f"{cmd[0]} failed ({res.returncode}):\n{res.stdout}\n{res.stderr}")
            os.replace(tmp, target)
        finally:
            fcntl.flock(lock, fcntl.LOCK_UN)
    return target


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))
    print(build_host(force="--force" in sys.argv))
