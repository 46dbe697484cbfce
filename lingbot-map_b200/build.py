"""Build the C-ABI library libgct_b200.so for sm_100a with nvcc and the PyTorch binding _gct_torch.so on top of it with
g++ (both in-tree, next to this file)."""
import os
import shutil
import subprocess
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
SOURCES = ["csrc/gct_attn_sm100.cu", "csrc/gct_elementwise.cu", "csrc/gct_manager.cu", "csrc/gct_static_scratch.cu",
           "csrc/gct_exchange.cu", "csrc/gct_decode.cu", "csrc/gct_render.cu"]
HEADERS = ["csrc/gct_common.h", "../include/gct_b200.h"]
LIB = os.path.join(HERE, "libgct_b200.so")
BINDING_SOURCE = "csrc/gct_torch.cpp"
BINDING = os.path.join(HERE, "_gct_torch.so")


def _nvcc():
    for cand in (os.environ.get("NVCC"), shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if cand and os.path.exists(cand):
            return cand
    raise RuntimeError("nvcc not found; set NVCC or put the CUDA toolkit on PATH")


def _older(target, sources):
    if not os.path.exists(target):
        return True
    t = os.path.getmtime(target)
    return any(os.path.getmtime(os.path.join(HERE, s)) > t for s in sources)


def _built_for():
    import torch
    return f"torch {torch.__version__}, Python {sys.version_info[0]}.{sys.version_info[1]}"


def binding_matches():
    """The binding in the tree was built for the torch and the Python that run now: it is linked against torch's C++ classes and
    Python's C API, and holds what it was built for as text."""
    if not os.path.exists(BINDING):
        return False
    with open(BINDING, "rb") as f:
        return f"binding built for {_built_for()};".encode() in f.read()


def _binding_needs_build():
    return _older(BINDING, [BINDING_SOURCE] + HEADERS) or not binding_matches()


def needs_build():
    return _older(LIB, SOURCES + HEADERS) or _binding_needs_build()


def _run(cmd, what):
    r = subprocess.run(cmd, cwd=HERE, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError(f"{what} failed:\n" + r.stdout + r.stderr)
    return r.stderr


def _build_binding():
    """The binding holds no device code; it finds libgct_b200.so beside itself ($ORIGIN)."""
    import sysconfig
    import torch
    from torch.utils import cpp_extension
    includes = cpp_extension.include_paths() + [sysconfig.get_paths()["include"], os.path.join(os.path.dirname(os.path.dirname(_nvcc())), "include")]
    torch_lib = os.path.join(os.path.dirname(torch.__file__), "lib")
    cmd = [os.environ.get("CXX", "g++"), "-O2", "-std=c++17", "-fPIC", "-shared", f"-D_GLIBCXX_USE_CXX11_ABI={int(torch.compiled_with_cxx11_abi())}",
           f'-DGCT_BUILT_FOR="{_built_for()}"']
    cmd += [x for i in includes for x in ("-isystem", i)]
    cmd += [BINDING_SOURCE, "-o", BINDING, f"-L{HERE}", "-l:libgct_b200.so", "-Wl,-rpath,$ORIGIN", f"-L{torch_lib}", "-ltorch", "-ltorch_cpu",
            "-ltorch_cuda", "-ltorch_python", "-lc10", "-lc10_cuda"]
    _run(cmd, "the C++ compiler")


def build(force=False, verbose=False):
    """Compile every source of the package into libgct_b200.so and _gct_torch.so.  Returns the library path."""
    if force or _older(LIB, SOURCES + HEADERS):
        cmd = [_nvcc(), "-O3", "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo",
               "-Xcompiler", "-fPIC", "-shared", "-cudart", "static", "-o", LIB] + SOURCES
        if verbose:
            cmd.insert(1, "-Xptxas=-v")
        log = _run(cmd, "nvcc")
        if verbose:
            print(log)
    if force or _binding_needs_build():
        _build_binding()
    return LIB


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))
