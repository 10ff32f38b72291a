"""Build libditto_b200.so (sm_100a only) in-tree with nvcc.

    python -m ditto_b200.build_lib            # rebuild if a source is newer than the library
    python -m ditto_b200.build_lib --force

nvcc cross-compiles without a GPU, so this also runs on a CPU-only machine.
"""
import os
import shutil
import subprocess
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
LIB_DIR = os.path.join(HERE, "lib")
LIB_PATH = os.path.join(LIB_DIR, "libditto_b200.so")
SOURCES = ["api.cu", "host_util.cu", "attention_sm100.cu", "attention_persistent_sm100.cu", "attention_narrow_sm100.cu", "attention_short_sm100.cu", "mlp_sm100.cu", "mlp_wide_sm100.cu", "mlp_pair_sm100.cu", "mlp_flow_sm100.cu", "mlp_tiles_sm100.cu", "mlp_waves_sm100.cu", "selftest_sm100.cu"]
# sources that are compiled in parts, an object and a GPU module each: (file, macro, number of parts)
IN_PARTS = [("mlp_tiles_kernel_sm100.cu", "DITTO_TILES_PART", 8), ("mlp_waves_kernel_sm100.cu", "DITTO_WAVES_PART", 8)]
NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
    "-Xcompiler", "-fPIC", "--use_fast_math",
]


def _nvcc():
    exe = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(exe):
        raise RuntimeError("nvcc not found; it is needed to build libditto_b200.so")
    return exe


def fastcall_path():
    """The operators' call path (csrc/fastcall.cpp).  torch's C++ interface is only good for the version that brings it, so
    the file's name says what it was compiled against: for another torch or Python there is no such file yet."""
    import torch
    return os.path.join(LIB_DIR, f"_fastcall-{torch.__version__}-cp{sys.version_info[0]}{sys.version_info[1]}.so")


def _stale():
    if not os.path.exists(LIB_PATH) or not os.path.exists(fastcall_path()):
        return True
    t = min(os.path.getmtime(LIB_PATH), os.path.getmtime(fastcall_path()))
    deps = [os.path.join(CSRC, f) for f in os.listdir(CSRC)]
    deps.append(os.path.join(HERE, "..", "include", "ditto_b200.h"))
    return any(os.path.getmtime(d) > t for d in deps if os.path.isfile(d))


def _fastcall_command():
    import sysconfig
    import torch
    from torch.utils import cpp_extension
    lib = os.path.join(os.path.dirname(torch.__file__), "lib")
    inc = [f"-I{p}" for p in cpp_extension.include_paths()]
    inc += [f"-I{sysconfig.get_paths()['include']}", f"-I{os.path.join(os.path.dirname(os.path.dirname(_nvcc())), 'include')}"]
    return ["g++", "-O2", "-std=c++17", "-shared", "-fPIC", f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
            *inc, os.path.join(CSRC, "fastcall.cpp"), "-o", fastcall_path(), f"-L{lib}", "-lc10", "-lc10_cuda", "-ltorch_cpu",
            "-ltorch_cuda", "-ltorch_python"]


def build(force=False, verbose=False):
    """Compile every CUDA source for sm_100a and link the shared library. Returns its path."""
    if not force and not _stale():
        return LIB_PATH
    os.makedirs(LIB_DIR, exist_ok=True)
    objs = []
    procs = []
    units = [(src, src.replace(".cu", ".o"), []) for src in SOURCES]
    units += [(src, src.replace(".cu", f"_{i}.o"), [f"-D{macro}={i}"]) for src, macro, n in IN_PARTS for i in range(n)]
    for src, name, defines in units:
        obj = os.path.join(LIB_DIR, name)
        cmd = [_nvcc(), *NVCC_FLAGS, *defines, "-c", os.path.join(CSRC, src), "-o", obj]
        if verbose:
            cmd.insert(1, "-Xptxas=-v")
        procs.append((src, subprocess.Popen(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)))
        objs.append(obj)
    procs.append(("fastcall.cpp", subprocess.Popen(_fastcall_command(), stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)))
    for src, p in procs:
        out, _ = p.communicate()
        if verbose and out:
            print(out)
        if p.returncode != 0:
            raise RuntimeError(f"compiling {src} failed:\n{out}")
    link = [_nvcc(), "-shared", "-o", LIB_PATH, *objs, "-lcudart"]
    r = subprocess.run(link, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)
    if r.returncode != 0:
        raise RuntimeError(f"link failed:\n{r.stdout}")
    return LIB_PATH


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))
