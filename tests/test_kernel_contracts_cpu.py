"""What the kernels' entry points accept and refuse, checked on the host before anything is launched."""

import glob
import os
import re
import shutil
import subprocess
import sys

import pytest
import torch

from axonn_b200.ops import _lib

native = pytest.mark.skipif(not (_lib.available() or shutil.which("nvcc")), reason="native library not built")


def _error():
    return _lib.lib().axb_last_error().decode()


@pytest.mark.parametrize("scale,ok", [(0.125, True), (1e-20, True), (0.0, False), (-0.125, False), (float("nan"), False),
                                      (float("inf"), False), (1e-42, False)])
@pytest.mark.parametrize("S", [77, 128])
def test_attention_kernels_take_positive_scales_only(S, scale, ok):
    """Masked scores are -inf before the softmax scale multiplies them: with zero the product is NaN and with a negative
    scale +inf.  Such calls belong to the general path, at every sequence length."""
    from axonn_b200.ops import attention_cuda

    qkv = torch.randn(1, S, 1, 3, 64).bfloat16()
    assert attention_cuda.supported(qkv, scale) is ok


@native
@pytest.mark.parametrize("scale", [0.0, -0.125, float("nan")])
def test_attention_entry_points_refuse_other_scales(scale):
    L, p = _lib.lib(), 4096                       # never dereferenced: the call is refused on the host
    assert L.axb_flash_attn_fwd(p, p, p, 1, 128, 1, 1, 64, scale, 0, None) == -1 and "scale" in _error()
    assert L.axb_flash_attn_bwd_split(p, p, p, p, p, p, 1, 128, 1, 1, 64, scale, 3, 0, None) == -1 and "scale" in _error()


@native
def test_prune_refuses_an_unaligned_workspace():
    """The scratch holds 64-bit words: 8-byte alignment is what the interface asks for (and all it needs)."""
    L = _lib.lib()
    assert L.axb_prune_topk(4096, 1 << 20, 0, 1000, 4096 + 4, 0, None) == -1 and "aligned" in _error()


@native
@pytest.mark.parametrize("which", range(6))
def test_norms_refuse_unaligned_operands(which):
    """The kernels move 16 bytes at a time (addresses that are never used: the call is refused on the host)."""
    L, p = _lib.lib(), [4096] * 6
    p[which] += 2
    assert L.axb_add_norm_fwd(*p, 4096, 4, 64, 64, 1e-5, 0, 0, 0, 0, None) == -1 and "aligned" in _error()
    dy, dres, x, gamma, dx, part = p
    assert L.axb_add_norm_bwd(dy, dres, x, gamma, 4096, dx, None, part, 4096, 4096, 4096, 4, 64, 64, 0, 0, 0, 0, 0, None) == -1
    assert "aligned" in _error()
    if which == 0:
        assert L.axb_colsum(dy, 4096, 4096, 4, 64, 0, 2, 0, None) == -1 and "aligned" in _error()


def test_every_status_code_of_the_kernels_has_a_name():
    """A wait that gave up is reported by name: every code that a kernel writes, and no code of a kernel that is gone."""
    csrc = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(_lib.__file__))), "csrc")
    text = "\n".join(open(f).read() for f in glob.glob(os.path.join(csrc, "*.cu*")))
    written = {int(c, 16) for c in re.findall(r"report_status\([^;]*?(0x[0-9a-f]{3})u\)", text)}
    assert len(written) > 20 and not written - set(_lib._STATUS_NAMES)
    mentioned = {int(c, 16) for c in re.findall(r"\b(0x[0-9a-f]{3})u?\b", text)}
    assert not set(_lib._STATUS_NAMES) - mentioned


@native
@pytest.mark.parametrize("name", ["AXONN_FA_FWD", "AXONN_NORM_WARP"])
def test_removed_switches_are_reported(name, monkeypatch):
    monkeypatch.setattr(_lib, "_LIB", None)
    monkeypatch.setenv(name, "0")
    with pytest.warns(UserWarning, match=name):
        _lib.lib()


@pytest.mark.parametrize("error", [ModuleNotFoundError("No module named 'torch'"), RuntimeError("g++ failed"), OSError("read-only")])
@pytest.mark.parametrize("built", [False, True])
def test_the_kernels_build_without_the_native_host_paths(error, built, monkeypatch, tmp_path):
    """The module of native host paths is optional: whatever keeps it from being built, the kernel library is."""
    from axonn_b200.utils import build

    def no_host(force=False):
        raise error

    def tool(cmd, **_):                               # what nvcc would write
        open(cmd[cmd.index("-o") + 1], "w").close()
        return subprocess.CompletedProcess(cmd, 0, "", "")
    monkeypatch.setattr(build, "LIB_DIR", str(tmp_path))
    monkeypatch.setattr(build, "OBJ_DIR", str(tmp_path / "obj"))
    monkeypatch.setattr(build, "LIB_PATH", str(tmp_path / "lib.so"))
    monkeypatch.setattr(build, "build_host", no_host)
    monkeypatch.setattr(build, "_nvcc", lambda: "nvcc")
    monkeypatch.setattr(build.subprocess, "run", tool)
    if built:
        open(build.LIB_PATH, "w").close()
    with pytest.warns(UserWarning, match=str(error).split()[0]):
        assert build.build_library(force=not built, verbose=False) == build.LIB_PATH
    assert os.path.exists(build.LIB_PATH)


def test_the_build_script_needs_no_torch():
    """The script imports nothing outside the standard library (the compile job has only Python and the CUDA toolkit)."""
    from axonn_b200.utils import build

    code = "import sys, runpy; sys.modules['torch'] = None; g = runpy.run_path(sys.argv[1]); g['_build_host_if_possible'](False)"
    r = subprocess.run([sys.executable, "-c", code, build.__file__], capture_output=True, text=True)
    assert r.returncode == 0 and "native host paths are not built" in r.stderr


@native
def test_native_host_paths_are_those_of_the_library(monkeypatch):
    """The module calls the launchers by address: it is used with the library whose header it was compiled against, and no other."""
    from axonn_b200.utils import build

    L = _lib.lib()
    if not os.path.exists(build.host_path()):
        pytest.skip("native host paths not built")
    assert f"-DAXB_INTERFACE={L.axb_interface() & 0xFFFFFFFF}u" == build._interface_flag()
    monkeypatch.setattr(_lib, "_HOST", _lib._UNSET)
    assert _lib.host() is not None

    class Older:                                      # another header's number, or a library from before there was one
        _name = "older.so"

        def __init__(self, **more):
            self.__dict__.update(more)

        def __getattr__(self, name):
            if name == "axb_interface":
                raise AttributeError(name)
            return getattr(L, name)
    for other in (Older(), Older(axb_interface=lambda: 1)):
        monkeypatch.setattr(_lib, "_HOST", _lib._UNSET)
        monkeypatch.setattr(_lib, "_LIB", other)
        with pytest.warns(UserWarning, match="another kernel library"):
            assert _lib.host() is None


def test_native_host_paths_are_rebuilt_with_the_header(monkeypatch, tmp_path):
    from axonn_b200.utils import build

    out, source, header = (str(tmp_path / n) for n in ("host.so", "host_ops.cpp", "axonn_b200.h"))
    for i, f in enumerate((source, out, header)):     # the header is the newest
        open(f, "w").close()
        os.utime(f, (100 + i, 100 + i))
    made = []

    def tool(cmd, **_):
        made.append(cmd)
        open(cmd[cmd.index("-o") + 1], "w").close()
        return subprocess.CompletedProcess(cmd, 0, "", "")
    monkeypatch.setattr(build, "HOST_SRC", source)
    monkeypatch.setattr(build, "HEADER", header)
    monkeypatch.setattr(build, "host_path", lambda: out)
    monkeypatch.setattr(build, "_nvcc", lambda: "/usr/local/cuda/bin/nvcc")
    monkeypatch.setattr(build.shutil, "which", lambda n: n)
    monkeypatch.setattr(build.subprocess, "run", tool)
    assert build.build_host() == out and len(made) == 1
    assert build.build_host() == out and len(made) == 1
