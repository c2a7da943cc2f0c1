"""Build libttt_mlp_b200.so (CUDA kernels + C ABI) in-tree with nvcc for sm_100a.

    python -m ttt_tk_b200.build            # rebuild if sources are newer than the library
    python -m ttt_tk_b200.build --force

nvcc cross-compiles without a GPU.  The library links only against cudart; the driver
entry point it needs (cuTensorMapEncodeTiled) is looked up at run time.
"""
import os
import shutil
import subprocess
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
LIB_DIR = os.path.join(HERE, "lib")
LIB_PATH = os.path.join(LIB_DIR, "libttt_mlp_b200.so")
SOURCES = ["ttt_capi.cu", "ttt_fwd_sm100.cu", "ttt_fwd_pair_sm100.cu", "ttt_bwd_sm100.cu", "ttt_bwd_pair_sm100.cu", "ttt_fwd_cluster_sm100.cu", "ttt_bwd_cluster_sm100.cu", "ttt_linear_fwd_sm100.cu", "ttt_linear_bwd_sm100.cu",
           "ttt_layout.cu", "ttt_glue.cu", "umma_selftest.cu"]
HEADERS = ["sm100_ptx.cuh", "ttt_device.cuh", "ttt_cluster.cuh", "ttt_internal.h", os.path.join("..", "..", "include", "ttt_mlp_b200.h")]
NVCC_FLAGS = ["-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
              "-shared", "-Xcompiler", "-fPIC", "-Xptxas", "-v"]


def _nvcc():
    for cand in (os.environ.get("NVCC"), shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if cand and os.path.exists(cand):
            return cand
    raise RuntimeError("nvcc not found (set NVCC)")


def needs_build():
    if not os.path.exists(LIB_PATH):
        return True
    t = os.path.getmtime(LIB_PATH)
    deps = [os.path.join(CSRC, s) for s in SOURCES + HEADERS]
    return any(os.path.getmtime(d) > t for d in deps)


def build(force=False, verbose=False):
    if not force and not needs_build():
        return LIB_PATH
    os.makedirs(LIB_DIR, exist_ok=True)
    cmd = [_nvcc()] + NVCC_FLAGS + ["-o", LIB_PATH] + SOURCES + ["-lcudart"]
    res = subprocess.run(cmd, cwd=CSRC, capture_output=True, text=True)
    if verbose or res.returncode != 0:
        sys.stderr.write(res.stdout + res.stderr)
    if res.returncode != 0:
        raise RuntimeError("nvcc failed building libttt_mlp_b200.so")
    with open(os.path.join(LIB_DIR, "ptxas.log"), "w") as f:
        f.write(res.stdout + res.stderr)
    return LIB_PATH


# ---------------------------------------------------------------------------------------------
# The PyTorch extension module `test_time_training` (the reference's module name): a C++ shim
# over the C ABI, built in-tree next to the library it links against.
EXT_NAME = "test_time_training"
EXT_SOURCE = os.path.join(CSRC, "test_time_training.cpp")


HOST_NAME = "_ttt_host"                      # validation and launch for ttt_tk_b200.ops
HOST_SOURCE = os.path.join(CSRC, "ttt_host.cpp")


def _module_path(name):
    import sysconfig
    return os.path.join(LIB_DIR, name + sysconfig.get_config_var("EXT_SUFFIX"))


def extension_path():
    return _module_path(EXT_NAME)


def _module_needs_build(source, out):
    """Missing, or older than its source or the C ABI's header, whose argument structs it fills."""
    deps = [source, os.path.join(CSRC, "..", "..", "include", "ttt_mlp_b200.h")]
    return not os.path.exists(out) or any(os.path.getmtime(d) > os.path.getmtime(out) for d in deps)


def _build_torch_module(name, source, out, force, verbose):
    """Compile one C++ module against the installed torch and the C-ABI library, with g++, in-tree."""
    build(force=False, verbose=verbose)
    if not force and not _module_needs_build(source, out):
        return out
    import sysconfig
    import torch
    from torch.utils import cpp_extension as ce
    inc = ce.include_paths(device_type="cuda") if "device_type" in ce.include_paths.__code__.co_varnames \
        else ce.include_paths(cuda=True)
    libdirs = ce.library_paths(device_type="cuda") if "device_type" in ce.library_paths.__code__.co_varnames \
        else ce.library_paths(cuda=True)
    cxx = os.environ.get("CXX", "g++")
    cmd = [cxx, "-O2", "-std=c++17", "-shared", "-fPIC", "-w",
           f"-DTORCH_EXTENSION_NAME={name}", "-DTORCH_API_INCLUDE_EXTENSION_H",
           f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
           "-I" + sysconfig.get_path("include")]
    cmd += ["-I" + p for p in inc]
    cmd += [source, "-o", out, "-L" + LIB_DIR, "-lttt_mlp_b200", "-Wl,-rpath,$ORIGIN"]
    cmd += ["-L" + p for p in libdirs] + ["-Wl,-rpath," + p for p in libdirs if "torch" in p]
    cmd += ["-lc10", "-lc10_cuda", "-ltorch_cpu", "-ltorch_cuda", "-ltorch", "-ltorch_python", "-lcudart"]
    res = subprocess.run(cmd, capture_output=True, text=True)
    if verbose or res.returncode != 0:
        sys.stderr.write(" ".join(cmd) + "\n" + res.stdout + res.stderr)
    if res.returncode != 0:
        raise RuntimeError(f"building the {name} extension failed")
    return out


def build_extension(force=False, verbose=False):
    """Compile ttt_tk_b200/lib/test_time_training*.so and ttt_tk_b200/lib/_ttt_host*.so."""
    _build_torch_module(HOST_NAME, HOST_SOURCE, _module_path(HOST_NAME), force, verbose)
    return _build_torch_module(EXT_NAME, EXT_SOURCE, extension_path(), force, verbose)


def _load(name, path):
    import importlib.util
    import torch  # noqa: F401  (libtorch must be loaded before the extension)
    spec = importlib.util.spec_from_file_location(name, path)
    mod = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(mod)
    return mod


def load_extension():
    """Import and return the `test_time_training` module (building it if needed)."""
    mod = _load(EXT_NAME, build_extension())
    sys.modules.setdefault(EXT_NAME, mod)
    return mod


def load_host():
    """Import and return the operators' native host side (building it, and the library, if it is out of date)."""
    path = _module_path(HOST_NAME)
    if _module_needs_build(HOST_SOURCE, path):
        _build_torch_module(HOST_NAME, HOST_SOURCE, path, False, False)
    return _load(HOST_NAME, path)


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose=True))
    print(build_extension())
