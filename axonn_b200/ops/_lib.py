"""Loader for the in-tree CUDA library (``axonn_b200/lib/libaxonn_b200.so``).

The kernels are plain ``extern "C"`` launchers compiled by nvcc for sm_100a
(see ``axonn_b200/utils/build.py``); they are called through ctypes with raw
device pointers and the current CUDA stream, so the library has no dependency
on the PyTorch C++ ABI; the host paths of calls that are bound by host time are
a module of their own, which has (``host``).  On a machine with a GPU a missing library is an error,
never a silent fallback.
"""

import ctypes
import os
import threading
import warnings

import torch

_LIB = None
_LOCK = threading.Lock()
LIB_DIR = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "lib")
# AXONN_LIB_PATH selects a library built elsewhere (e.g. an ablation build with -DAXB_ABLATION);
# AXONN_DEBUG_BOUNDS=1 selects the bounds-checking build when it has been built
# (``python axonn_b200/utils/build.py --debug-bounds``)
_DEBUG_LIB = os.path.join(LIB_DIR, "libaxonn_b200_debug.so")
LIB_PATH = os.environ.get("AXONN_LIB_PATH") or (
    _DEBUG_LIB if os.environ.get("AXONN_DEBUG_BOUNDS", "0") not in ("", "0") and os.path.exists(_DEBUG_LIB)
    else os.path.join(LIB_DIR, "libaxonn_b200.so"))

# Kernels launched through this library since the last reset are ``launch_count`` (see ``__getattr__``): those counted here and
# those of the native host paths.
_launches = 0
_HOST = _UNSET = object()
_HOST_LAUNCHERS = ("axb_norm_fwd", "axb_norm_bwd", "axb_add_norm_fwd", "axb_add_norm_bwd", "axb_norm_grid", "axb_gemm",
                   "axb_flash_attn_fwd", "axb_last_error")


def __getattr__(name):
    if name == "launch_count":
        return _launches + (_HOST.launches() if _HOST is not _UNSET and _HOST is not None else 0)
    raise AttributeError(f"module {__name__!r} has no attribute {name!r}")


class KernelError(RuntimeError):
    pass


# Argument types of the launchers that run once per layer (i int, l long long, f float, p pointer).  With them declared,
# plain Python numbers and addresses are converted by ctypes itself; without, every call builds an object per argument
# (some fifteen of them for a GEMM).
_SIGNATURES = {
    "axb_gemm": "ippppp" "iiiiiiii" "p",
    "axb_gemm_swiglu": "i" "pppp" "iiii" "p" "iii" "p",
    "axb_gemm_on_pairs": "iii",
    "axb_gemm_dgelu": "ppppp" "iiii" "p",
    "axb_fold_columns": "pp" "iii" "p",
    "axb_gemm_ce_pays": "iiii",
    "axb_gemm_ce": "pppp" "iiii" "p",
    "axb_ce_fwd_parts": "ppppppp" "ii" "l" "p",
    "axb_norm_fwd": "ppppp" "iii" "f" "iiii" "p",
    "axb_norm_bwd": "pppppppppp" "iiiiiiii" "p",
    "axb_add_norm_fwd": "ppppppp" "iii" "f" "iiii" "p",
    "axb_add_norm_bwd": "ppppppppppp" "iiiiiiii" "p",
    "axb_norm_grid": "ii",
    "axb_colsum_splits": "iii",
    "axb_colsum": "ppp" "iiiii" "p",
    "axb_gelu_bwd_colsum": "ppppp" "iiiii" "p",
    "axb_gelu_fwd": "pplp",
    "axb_gelu_bwd": "ppplp",
    "axb_swiglu_fwd": "ppiip",
    "axb_swiglu_bwd": "pppiip",
    "axb_rope": "pp" "l" "iiii" "l" "i" "p",
    "axb_flash_attn_fwd": "ppp" "iiiii" "f" "i" "p",
    "axb_flash_attn_bwd_split": "pppppp" "iiiii" "f" "ii" "p",
    "axb_flash_attn_bwd_scratch": "iii",
    "axb_ce_fwd_mean": "pppppp" "ii" "l" "p",
    "axb_ce_bwd": "pppp" "iii" "l" "p",
    "axb_multi_l2norm_sq": "p" "il" "pp",
    "axb_multi_clip_factor": "p" "il" "f" "pp",
    "axb_multi_scale": "p" "il" "pp",
    "axb_multi_adamw": "p" "il" "fffffff" "ppp",
    "axb_moe_route": "piiiii" "ppppppppppp" "p",
    "axb_moe_route_bwd": "piii" "pppppp" "p",
    "axb_prune_topk": "p" "lil" "p" "i" "p",
}
# Switches of kernels that are gone.  The one kernel that is left covers what they selected; a program that still sets
# one is told so instead of being ignored.
_REMOVED_SWITCHES = {
    "AXONN_FA_FWD": "the two-tile attention forward serves every sequence length",
    "AXONN_NORM_WARP": "the ring kernel is the norm forward for every hidden size up to 8192",
}
_CTYPES = {"i": ctypes.c_int, "l": ctypes.c_longlong, "f": ctypes.c_float, "p": ctypes.c_void_p}


def available() -> bool:
    return os.path.exists(LIB_PATH)


def lib():
    """Return the loaded library, building it first when it is missing and nvcc
    is present."""
    global _LIB
    if _LIB is not None:
        return _LIB
    with _LOCK:
        if _LIB is None:
            if not os.path.exists(LIB_PATH):
                from ..utils import build

                build.build_library(verbose=False)
            L = ctypes.CDLL(LIB_PATH, mode=ctypes.RTLD_GLOBAL)
            L.axb_last_error.restype = ctypes.c_char_p
            for name, sig in _SIGNATURES.items():
                if hasattr(L, name):
                    getattr(L, name).argtypes = [_CTYPES[c] for c in sig]
            L.axb_flash_attn_bwd_scratch.restype = ctypes.c_longlong
            ms = os.environ.get("AXONN_COMM_TIMEOUT_MS")
            if ms:
                L.axb_set_wait_timeout_ms(ctypes.c_uint(int(ms)))
            _LIB = L      # published when complete: another thread may be waiting for it without the lock
            for name, why in _REMOVED_SWITCHES.items():
                if name in os.environ:
                    warnings.warn(f"{name} has no effect: {why}", stacklevel=2)
    return _LIB


def host():
    """The native host paths (``csrc/host_ops.cpp``), bound to the loaded library; ``None`` where they have not been built for this
    PyTorch (or ``AXONN_HOST_OPS=0``): the Python code beside every use of them launches the same kernels."""
    return _HOST if _HOST is not _UNSET else _load_host()


def _load_host():
    global _HOST
    L = lib()
    with _LOCK:
        if _HOST is _UNSET:
            import importlib.util

            from ..utils.build import host_path

            path, module = host_path(), None
            if os.environ.get("AXONN_HOST_OPS", "1") != "0" and os.path.exists(path):
                spec = importlib.util.spec_from_file_location("axonn_host", path)
                launchers = {n: ctypes.cast(getattr(L, n), ctypes.c_void_p).value for n in _HOST_LAUNCHERS if hasattr(L, n)}
                interface = L.axb_interface() & 0xFFFFFFFF if hasattr(L, "axb_interface") else 0
                try:
                    module = importlib.util.module_from_spec(spec)
                    spec.loader.exec_module(module)
                    why = "" if module.bind(launchers, KernelError, torch.nn.Parameter, interface) else "built for another kernel library"
                except (ImportError, RuntimeError) as e:
                    why = str(e)
                if why:
                    warnings.warn(f"the native host paths are not used ({why}); rebuild them (axonn_b200/utils/build.py)", stacklevel=2)
                    module = None
            _HOST = module
    return _HOST


def set_wait_timeout_ms(ms: int):
    """Deadline of every device-side wait (mbarrier, peer flag).  A kernel whose wait runs out returns and
    reports through the status word (``check_status``).  Default 120000 ms; ``AXONN_COMM_TIMEOUT_MS`` sets it
    at load time."""
    lib().axb_set_wait_timeout_ms(ctypes.c_uint(int(ms)))


def use_cuda_kernels(*tensors) -> bool:
    """True when the operands live on a GPU (then the library is mandatory)."""
    return len(tensors) > 0 and all(t is None or t.is_cuda for t in tensors) and any(
        t is not None for t in tensors)


def stream_ptr() -> ctypes.c_void_p:
    return ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)


def stream() -> int:
    """Address of the current CUDA stream of the current device, for launchers with declared argument types."""
    return torch._C._cuda_getCurrentRawStream(torch._C._cuda_getDevice())


def addr(t):
    """Device address of ``t`` (``None``: null), for launchers with declared argument types."""
    return None if t is None else t.data_ptr()


def ptr(t) -> ctypes.c_void_p:
    return ctypes.c_void_p(0 if t is None else t.data_ptr())


def check(status: int, what: str):
    global _launches
    if status != 0:
        msg = lib().axb_last_error()
        raise KernelError(f"{what} failed (status {status}): {msg.decode() if msg else ''}")
    _launches += 1


def add_launches(n: int):
    global _launches
    _launches += n


def reset_launch_count():
    global _launches
    _launches = -_HOST.launches() if _HOST is not _UNSET and _HOST is not None else 0


_STATUS_NAMES = {
    0x101: "GEMM producer: shared-memory stage never freed",
    0x102: "GEMM MMA issuer: operand stage or accumulator never arrived",
    0x104: "GEMM epilogue: accumulator never completed",
    0x108: "fused GEMM: a peer never finished the previous call on this buffer",
    0x110: "all-gather stage: a peer never published its weight shard",
    0x120: "fused reduction: aborted while waiting for partial tiles",
    0x121: "fused reduction: partial tiles of a peer never arrived",
    0x122: "fused reduction (shared-memory ring): inbox slots never arrived",
    0x123: "fused reduction (shared-memory ring): ring group never freed",
    0x109: "fused all-reduce (two-shot): a peer never finished writing its rows of the result",
    0x124: "fused all-reduce (two-shot): a peer never announced where its output lies",
    0x201: "expert dispatch / combine: a peer never signalled",
    0x301: "gradient all-reduce: a peer never published its bucket",
    0x302: "gradient all-reduce: a peer never delivered its partial slices",
    0x303: "gradient all-reduce: a peer never delivered its reduced slice",
    0x501: "row all-to-all: a peer never announced its output",
    0x502: "row all-to-all / embedding rows: a peer never finished",
    0x503: "embedding row fetch: a peer never published its table shard",
    0x504: "embedding gradient: a peer never published its gradient shard",
    0x701: "bounds check (debug build): inbox slot outside the peer's inbox",
    0x702: "bounds check (debug build): output element outside C",
    0x703: "bounds check (debug build): flag index outside the flag array",
    0x405: "flash attention forward: producer timed out",
    0x406: "flash attention forward: MMA issuer timed out",
    0x407: "flash attention forward: softmax warps timed out",
    0x411: "flash attention backward (one kernel): producer timed out",
    0x412: "flash attention backward (one kernel): MMA issuer timed out",
    0x414: "flash attention backward (one kernel): softmax / reduction warps timed out",
    0x421: "flash attention backward, dQ kernel: producer timed out",
    0x422: "flash attention backward, dQ kernel: score MMA issuer timed out",
    0x423: "flash attention backward, dQ kernel: softmax warps timed out",
    0x424: "flash attention backward, dQ kernel: dQ MMA issuer timed out",
    0x431: "flash attention backward, dK / dV kernel: producer timed out",
    0x432: "flash attention backward, dK / dV kernel: MMA issuer timed out",
    0x433: "flash attention backward, dK / dV kernel: softmax warps timed out",
    0x151: "split-K GEMM producer timed out",
    0x152: "split-K GEMM MMA issuer timed out",
    0x154: "split-K GEMM epilogue timed out",
    0x141: "CTA-pair GEMM producer timed out",
    0x142: "CTA-pair GEMM MMA issuer timed out",
    0x144: "CTA-pair GEMM epilogue timed out",
}


class AxonnCommTimeout(KernelError):
    """A device-side wait (mbarrier or peer flag) ran into its deadline; ``status`` is the kernel's reason code."""

    def __init__(self, status: int):
        self.status = status
        super().__init__(f"device-side wait timed out (status 0x{status:x}: {_STATUS_NAMES.get(status, 'unknown')})")


def device_status(device=None, clear=True) -> int:
    """Status word that kernels write when one of their bounded waits gave up (0: none did).  The word lives
    in mapped host memory, so reading it needs no synchronisation; it is meaningful once the kernels in
    question have finished (e.g. after reading the loss)."""
    import torch

    if not available() or not torch.cuda.is_available():
        return 0
    dev = torch.cuda.current_device() if device is None else int(device)
    return int(lib().axb_device_status(ctypes.c_int(dev), ctypes.c_int(1 if clear else 0)))


def check_status(device=None):
    """Raise ``AxonnCommTimeout`` (a ``KernelError``) if a kernel on ``device`` reported a timed-out wait since
    the last check."""
    st = device_status(device, clear=True)
    if st not in (0, 0xFFFFFFFF):
        raise AxonnCommTimeout(st)
