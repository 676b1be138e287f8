"""Build the in-tree CUDA library for sm_100a.

``build_library()`` compiles every ``csrc/*.cu`` with
``nvcc -gencode arch=compute_100a,code=sm_100a -lineinfo`` (object files in
parallel, then one link) into ``axonn_b200/lib/libaxonn_b200.so``.  nvcc
cross-compiles without a GPU.  The library is rebuilt only when a source or
header is newer than it.  With it goes the module of native host paths, which
wants PyTorch's headers and g++: where it cannot be built there is a warning, and
the Python code launches the same kernels.
"""

import glob
import os
import shutil
import subprocess
import sys
import warnings
import zlib
from concurrent.futures import ThreadPoolExecutor

PKG = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(PKG, "csrc")
LIB_DIR = os.path.join(PKG, "lib")
OBJ_DIR = os.path.join(LIB_DIR, "obj")
LIB_PATH = os.path.join(LIB_DIR, "libaxonn_b200.so")
HOST_SRC = os.path.join(CSRC, "host_ops.cpp")
HEADER = os.path.join(CSRC, "axonn_b200.h")

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
    "--use_fast_math", "-Xcompiler", "-fPIC", "-Xptxas", "-v",
]


def _nvcc():
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        raise RuntimeError("nvcc not found: cannot build axonn_b200's CUDA library")
    return nvcc


def sources():
    return sorted(glob.glob(os.path.join(CSRC, "*.cu")))


def _newest_input():
    files = sources() + glob.glob(os.path.join(CSRC, "*.cuh")) + glob.glob(os.path.join(CSRC, "*.h"))
    return max(os.path.getmtime(f) for f in files)


def up_to_date():
    return os.path.exists(LIB_PATH) and os.path.getmtime(LIB_PATH) >= _newest_input()


def _interface_flag():
    """What the library and the module of native host paths are told of the header that both are compiled against."""
    with open(HEADER, "rb") as f:
        return f"-DAXB_INTERFACE={zlib.crc32(f.read())}u"


def host_path():
    """Where the native host paths are for this PyTorch and this Python, whose C++ interfaces they use."""
    import torch

    return os.path.join(LIB_DIR, f"axonn_host-{torch.__version__}-{sys.implementation.cache_tag}.so")


def build_host(force=False):
    """The native host paths (``csrc/host_ops.cpp``): a Python module against PyTorch's C++ API, without device code."""
    out = host_path()
    if not force and os.path.exists(out) and os.path.getmtime(out) >= max(map(os.path.getmtime, (HOST_SRC, HEADER))):
        return out
    import sysconfig

    import torch

    gxx = shutil.which("g++")
    if gxx is None:
        raise RuntimeError("g++ not found: cannot build axonn_b200's native host paths")
    root = os.path.dirname(torch.__file__)
    cuda = os.path.dirname(os.path.dirname(os.path.realpath(_nvcc())))
    dirs = [os.path.join(root, "include"), os.path.join(root, "include", "torch", "csrc", "api", "include"),
            sysconfig.get_paths()["include"], os.path.join(cuda, "include")]
    cmd = [gxx, "-O2", "-std=c++17", "-fPIC", "-shared", f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}"]
    cmd += [_interface_flag()] + ["-I" + d for d in dirs + [CSRC]] + [HOST_SRC, "-o", out + ".tmp", "-L" + os.path.join(root, "lib")]
    cmd += ["-lc10", "-lc10_cuda", "-ltorch_cpu", "-ltorch_python"]
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError(f"g++ failed for {HOST_SRC}:\n{r.stdout}\n{r.stderr}")
    os.replace(out + ".tmp", out)
    return out


def _build_host_if_possible(force):
    """The native host paths are optional: the kernels neither need them nor PyTorch."""
    try:
        build_host(force)
    except (ImportError, OSError, RuntimeError) as e:
        warnings.warn(f"the native host paths are not built, the Python code launches the kernels instead: {e}", stacklevel=3)


def _compile(src, verbose):
    obj = os.path.join(OBJ_DIR, os.path.basename(src)[:-3] + ".o")
    hdr_time = max([os.path.getmtime(f) for f in glob.glob(os.path.join(CSRC, "*.cuh")) +
                    glob.glob(os.path.join(CSRC, "*.h"))] + [0])
    if os.path.exists(obj) and os.path.getmtime(obj) >= max(os.path.getmtime(src), hdr_time):
        return obj, ""
    cmd = [_nvcc()] + NVCC_FLAGS + [_interface_flag(), "-I", CSRC, "-c", src, "-o", obj]
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError(f"nvcc failed for {src}:\n{r.stdout}\n{r.stderr}")
    return obj, r.stderr


def build_variant(out_path, extra_flags, obj_dir):
    """Build a variant of the library (extra nvcc flags, e.g. ``-DAXB_ABLATION``) to ``out_path``; select it
    at run time with ``AXONN_LIB_PATH``.  The default library is not touched."""
    os.makedirs(obj_dir, exist_ok=True)
    objs = []
    for src in sources():
        obj = os.path.join(obj_dir, os.path.basename(src)[:-3] + ".o")
        r = subprocess.run([_nvcc()] + NVCC_FLAGS + list(extra_flags) + [_interface_flag(), "-I", CSRC, "-c", src, "-o", obj],
                           capture_output=True, text=True)
        if r.returncode != 0:
            raise RuntimeError(f"nvcc failed for {src}:\n{r.stdout}\n{r.stderr}")
        objs.append(obj)
    r = subprocess.run([_nvcc(), "-shared", "-o", out_path] + objs + ["-gencode", "arch=compute_100a,code=sm_100a"],
                       capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError(f"link failed:\n{r.stdout}\n{r.stderr}")
    return out_path


def build_library(force=False, verbose=True):
    if not force and up_to_date():
        _build_host_if_possible(force)
        return LIB_PATH
    os.makedirs(OBJ_DIR, exist_ok=True)
    with ThreadPoolExecutor(max_workers=min(8, os.cpu_count() or 2)) as ex:
        host = ex.submit(_build_host_if_possible, force)
        results = list(ex.map(lambda s: _compile(s, verbose), sources()))
    objs = [o for o, _ in results]
    log = "\n".join(l for _, l in results if l)
    with open(os.path.join(LIB_DIR, "ptxas.log"), "a") as f:
        f.write(log)
    cmd = [_nvcc(), "-shared", "-o", LIB_PATH + ".tmp"] + objs + ["-gencode", "arch=compute_100a,code=sm_100a"]
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError(f"link failed:\n{r.stdout}\n{r.stderr}")
    os.replace(LIB_PATH + ".tmp", LIB_PATH)
    if verbose:
        print(f"built {LIB_PATH} from {len(objs)} sources", file=sys.stderr)
    host.result()                  # what is not one of the reasons to do without is an error, after the library is there
    return LIB_PATH


DEBUG_LIB_PATH = os.path.join(LIB_DIR, "libaxonn_b200_debug.so")


def build_debug_library():
    """The bounds-checking build (``-DAXB_DEBUG_BOUNDS``): kernels verify computed offsets into peer memory
    before every store and record violations in the device status word instead of making the access.  Loaded
    instead of the normal library when ``AXONN_DEBUG_BOUNDS=1`` and the file exists."""
    os.makedirs(LIB_DIR, exist_ok=True)
    return build_variant(DEBUG_LIB_PATH, ["-DAXB_DEBUG_BOUNDS"], os.path.join(LIB_DIR, "obj_debug"))


SANITIZER_LIB_PATH = os.path.join(LIB_DIR, "libaxonn_b200_asan.so")


def build_sanitizer_library():
    """The host code of the library (allocators, symmetric heap, launch wrappers, status handling) compiled with
    AddressSanitizer and UndefinedBehaviorSanitizer; device code is unchanged.  Run the CPU tests against it with

        AXONN_LIB_PATH=<this file> LD_PRELOAD="$(gcc -print-file-name=libasan.so) $(gcc -print-file-name=libubsan.so)" \
        ASAN_OPTIONS=detect_leaks=0:abort_on_error=1 UBSAN_OPTIONS=halt_on_error=1 \
        python -m pytest tests/test_arena_cpu.py tests/test_symm_heap_cpu.py tests/test_ops_cpu.py

    (leak detection is off because the Python interpreter itself never frees everything)."""
    os.makedirs(LIB_DIR, exist_ok=True)
    flags = ["-Xcompiler", "-fsanitize=address", "-Xcompiler", "-fsanitize=undefined", "-Xcompiler",
             "-fno-omit-frame-pointer"]
    return build_variant(SANITIZER_LIB_PATH, flags, os.path.join(LIB_DIR, "obj_asan"))


if __name__ == "__main__":
    if "--debug-bounds" in sys.argv:
        print(build_debug_library())
    elif "--sanitize" in sys.argv:
        print(build_sanitizer_library())
    else:
        build_library(force="--force" in sys.argv)
