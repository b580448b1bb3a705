"""In-tree build of the native parts: ``python -m flashkda_b200.build``.

``libflashkda_b200.so``: the CUDA library behind the C ABI, plain ``nvcc`` for sm_100a only, no third-party headers.
``_host.so``: the host side of ``fwd`` (argument checks, scratch, the call of the C ABI), a CPython extension against the
installed PyTorch's headers, plain ``g++``.  Both sit next to this file (git-ignored).
"""
import glob
import os
import subprocess
import sys
import sysconfig

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
LIB = os.path.join(HERE, "libflashkda_b200.so")
HOST_SRC = os.path.join(CSRC, "fkda_host.cpp")
HOST = os.path.join(HERE, "_host.so")

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
    "-ftz=true",  # the reference is built with --use_fast_math; only its flush-to-zero part is numerically
                  # visible in the instruction sequences used here
    "-Xcompiler", "-fPIC", "-shared", "-Xlinker", "-soname=libflashkda_b200.so",
]


def sources():
    return sorted(glob.glob(os.path.join(CSRC, "*.cu")))


def _stale(target, deps) -> bool:
    if not os.path.exists(target):
        return True
    t = os.path.getmtime(target)
    return any(os.path.getmtime(d) > t for d in deps)


def _headers():
    return glob.glob(os.path.join(HERE, "..", "include", "*.h"))


def needs_build() -> bool:
    return _stale(LIB, sources() + glob.glob(os.path.join(CSRC, "*.cuh")) + glob.glob(os.path.join(CSRC, "*.h")) + _headers())


def _run(cmd, what, verbose):
    env = dict(os.environ)
    env.pop("CC", None)
    env.pop("CXX", None)
    res = subprocess.run(cmd, env=env, capture_output=True, text=True)
    if verbose or res.returncode != 0:
        sys.stderr.write(res.stdout + res.stderr)
    if res.returncode != 0:
        raise RuntimeError("the compiler failed building " + what)


def _host_command():
    import torch
    root = os.path.dirname(torch.__file__)
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    inc = [os.path.join(root, "include"), os.path.join(root, "include", "torch", "csrc", "api", "include"),
           os.path.join(cuda, "include"), sysconfig.get_paths()["include"]]
    abi = int(torch._C._GLIBCXX_USE_CXX11_ABI)
    return (["g++", "-O2", "-std=c++17", "-fPIC", "-shared", f"-D_GLIBCXX_USE_CXX11_ABI={abi}"] +
            [x for d in inc for x in ("-isystem", d)] + ["-o", HOST, HOST_SRC, LIB, "-L" + os.path.join(root, "lib"),
             "-ltorch_python", "-ltorch_cpu", "-lc10", "-lc10_cuda", "-Wl,-rpath,$ORIGIN"])


def build(force: bool = False, verbose: bool = False) -> str:
    if force or needs_build():
        nvcc = os.environ.get("NVCC", "nvcc")
        _run([nvcc] + NVCC_FLAGS + (["-Xptxas", "-v"] if verbose else []) + ["-o", LIB] + sources(),
             "libflashkda_b200.so", verbose)
    if force or _stale(HOST, [HOST_SRC, LIB] + _headers()):
        _run(_host_command(), "_host.so", verbose)
    return LIB


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))
