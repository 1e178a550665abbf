"""Builds the two native libraries in-tree (no JIT cache, no torch extension machinery):

    libquamba_b200.so    the kernels behind the C ABI, nvcc for sm_100a
    _native.<tag>.so     the host path (CPython extension over torch's C++ API), g++; the tag is the interpreter's

    python -m quamba_b200.build            # rebuilds what is out of date

An object is out of date when a file it is made of is newer, or when the command that would make it is not the one that did: the
host path's names the interpreter's and torch's headers and torch's version.
"""
import os
import subprocess
import sys
import sysconfig
from pathlib import Path

PKG = Path(__file__).resolve().parent
CSRC = PKG / "csrc"
LIB = PKG / "libquamba_b200.so"
NATIVE = PKG / ("_native" + sysconfig.get_config_var("EXT_SUFFIX"))
SOURCES = ["lib.cu", "conv1d.cu", "hadamard.cu", "hadamard_tc.cu", "sscan.cu", "sscan_cl.cu", "ssd.cu", "ssd_tc.cu", "linear.cu", "gemm_tc.cu", "norm.cu",
           "embedding.cu", "decode.cu", "peer.cu"]
NATIVE_SOURCES = ["binding.cpp", "binding_layers.cpp"]
NVCC_FLAGS = ["-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17", "-lineinfo",
              "-Xcompiler", "-fPIC", "--expt-relaxed-constexpr", "-Xptxas", "-v"]
CUDA = Path(os.environ.get("CUDA_HOME", "/usr/local/cuda"))


def _command_file(obj: Path) -> Path:
    return obj.with_suffix(".cmd")


def _stale(obj: Path, src: Path, cmd) -> bool:
    if not obj.exists() or not _command_file(obj).exists() or _command_file(obj).read_text() != " ".join(cmd):
        return True
    t = obj.stat().st_mtime
    headers = list(CSRC.glob("*.cuh")) + list(CSRC.glob("*.inc")) if src.suffix == ".cu" else list(CSRC.glob("*.h"))
    return any(d.stat().st_mtime > t for d in [src, PKG.parent / "include" / "quamba_b200.h"] + headers)


def _older(target: Path, objs) -> bool:
    return not target.exists() or any(Path(o).stat().st_mtime > target.stat().st_mtime for o in objs)


def _native_flags():
    import torch
    inc = Path(torch.__file__).parent / "include"
    dirs = [inc, inc / "torch" / "csrc" / "api" / "include", CUDA / "include", sysconfig.get_paths()["include"]]
    return ["-O2", "-std=c++17", "-fPIC", "-fvisibility=hidden", f'-DQBN_TORCH_VERSION="{torch.__version__}"', f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
            *[f for d in dirs for f in ("-isystem", str(d))]], Path(torch.__file__).parent / "lib"


def build(verbose: bool = False, force: bool = False) -> Path:
    nvcc = os.environ.get("NVCC", str(CUDA / "bin" / "nvcc"))
    cxx = os.environ.get("CXX", "g++")
    objdir = PKG / "build"
    objdir.mkdir(exist_ok=True)
    flags, torch_lib = _native_flags()
    procs = []
    for name in SOURCES + NATIVE_SOURCES:
        src, obj = CSRC / name, objdir / (name + ".o")
        cmd = [nvcc, *NVCC_FLAGS] if src.suffix == ".cu" else [cxx, *flags]
        if force or _stale(obj, src, cmd):
            _command_file(obj).unlink(missing_ok=True)
            procs.append((name, cmd, subprocess.Popen([*cmd, "-c", str(src), "-o", str(obj)], stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)))
    failed = False
    for name, cmd, p in procs:
        out, _ = p.communicate()
        if p.returncode == 0:
            _command_file(objdir / (name + ".o")).write_text(" ".join(cmd))
        if verbose or p.returncode != 0:
            sys.stderr.write(f"--- {name} ---\n{out}\n")
        (objdir / (name + ".log")).write_text(out)
        failed |= p.returncode != 0
    if failed:
        raise RuntimeError("compilation failed; see the log above")
    kernels, native = ([str(objdir / (n + ".o")) for n in names] for names in (SOURCES, NATIVE_SOURCES))
    if _older(LIB, kernels):
        subprocess.run([nvcc, "-shared", "-o", str(LIB), *kernels, "-gencode", "arch=compute_100a,code=sm_100a"], check=True)
    (PKG / "_native.so").unlink(missing_ok=True)             # an untagged one would be loaded by any interpreter
    if _older(NATIVE, native):
        subprocess.run([cxx, "-shared", "-o", str(NATIVE), *native, f"-L{PKG}", "-l:libquamba_b200.so",
                        f"-L{torch_lib}", "-ltorch_python", "-ltorch", "-ltorch_cpu", "-ltorch_cuda", "-lc10", "-lc10_cuda", "-Wl,-rpath,$ORIGIN"],
                       check=True)
    return LIB


if __name__ == "__main__":
    print(build(verbose="-v" in sys.argv, force="-f" in sys.argv))
