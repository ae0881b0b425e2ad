"""The launcher extension's argument passing (csrc/launcher.c) and calls of autograd functions without gradients."""
import ctypes
import importlib.util
import subprocess

import pytest
import torch
from torch.autograd import forward_ad

from atorch_b200 import build
from atorch_b200.ops.function import call

C_SOURCE = r"""
#include <string.h>
static double seen[64];
const double* last(void) { return seen; }
int mixed(void* a, const void* b, int c, long long d, float e, int g, void* h, long long i, int j, float k, int l, int m,
          const int* n, int o, long long p, float q, int r, long long s, int t, int u) {
  const double v[] = {(double)(long long)a, (double)(long long)b, c, (double)d, e, g, (double)(long long)h, (double)i, j, k,
                      l, m, n[0], n[1], o, (double)p, q, r, (double)s, t, u};
  memcpy(seen, v, sizeof(v));
  return -7;
}
"""


def _module(tmp_path):
    build._build_launcher(False)
    spec = importlib.util.spec_from_file_location("_launcher", build.LAUNCHER)
    launcher = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(launcher)
    (tmp_path / "callee.c").write_text(C_SOURCE)
    subprocess.run(["gcc", "-O2", "-shared", "-fPIC", str(tmp_path / "callee.c"), "-o", str(tmp_path / "callee.so")], check=True)
    lib = ctypes.CDLL(str(tmp_path / "callee.so"))
    lib.last.restype = ctypes.POINTER(ctypes.c_double)
    return launcher, lib, launcher.Launcher(ctypes.cast(lib.mixed, ctypes.c_void_p).value, "ppilfiplifiipilfilii")


def test_arguments_in_registers_and_on_the_stack(tmp_path):
    """Integers of both widths, pointers in every form and floats between them, more than the registers hold; numbers are cut
    to the declared width like ctypes does; wrong counts and types are errors and call nothing."""
    launcher, lib, fn = _module(tmp_path)
    arr = (ctypes.c_int * 2)(21, -22)
    args = (1 << 40, None, -3, -(1 << 40), 1.5, True, ctypes.c_void_p(0), 7, (1 << 33) | 5, 2, ctypes.c_int(9), -11, arr, -1,
            (1 << 50) + 1, ctypes.c_float(0.25), 13, -14, -15, 16)
    before = launcher.count()
    assert fn(*args) == -7
    assert lib.last()[:21] == [1 << 40, 0, -3, -(1 << 40), 1.5, 1, 0, 7, 5, 2, 9, -11, 21, -22, -1, (1 << 50) + 1, 0.25, 13,
                               -14, -15, 16]
    assert launcher.count() == before + 1
    for bad in (args[:-1], args + (1,), ("x",) + args[1:], args[:2] + (1.5,) + args[3:], args[:4] + (None,) + args[5:]):
        with pytest.raises((TypeError, AttributeError)):
            fn(*bad)
    assert launcher.count() == before + 1
    with pytest.raises(ValueError):
        launcher.Launcher(1, "px")


def test_launcher_belongs_to_one_python(tmp_path, monkeypatch):
    """Its name says to which; it appears whole; what is left where it cannot be built is ctypes, with the same calls."""
    import sysconfig

    from atorch_b200 import _lib

    assert build.LAUNCHER.name == "_launcher" + sysconfig.get_config_var("EXT_SUFFIX")
    launcher, lib, _ = _module(tmp_path)
    monkeypatch.setattr(build, "OUT_DIR", tmp_path)
    monkeypatch.setattr(build, "LAUNCHER", tmp_path / build.LAUNCHER.name)
    monkeypatch.setenv("CC", "false")
    with pytest.warns(UserWarning, match="ctypes"):
        assert not build.build_launcher()
    with pytest.warns(UserWarning, match="ctypes"):
        assert _lib._load_launcher() is None
    assert not list(tmp_path.glob("_launcher*"))
    monkeypatch.setitem(_lib.SIGNATURES, "mixed", "ppilfiplifiipilfilii")
    monkeypatch.setattr(_lib, "_ctypes_launches", 0)
    arr = (ctypes.c_int * 2)(21, -22)
    args = (1 << 40, None, -3, -(1 << 40), 1.5, True, None, 7, 5, 2.0, 9, -11, ctypes.addressof(arr), -1, 1 << 50, 0.25, 13, -14,
            -15, 16)
    seen = []
    for module in (launcher, None):
        assert _lib._CountingLib(lib, module).mixed(*args) == -7
        seen.append(lib.last()[:21])
    assert seen[0] == seen[1] and _lib._ctypes_launches == 1
    monkeypatch.delenv("CC")
    assert build.build_launcher() and [f.name for f in tmp_path.glob("_launcher*")] == [build.LAUNCHER.name]


class _Double(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x):
        ctx.save_for_backward(x)
        ctx.seen = ctx.needs_input_grad
        _Double.last = tuple(ctx.needs_input_grad)
        return x * 2

    @staticmethod
    def backward(ctx, g):
        return g * 2


def test_call_without_gradients():
    """With gradients on, the node; off, the forward alone, which is told that nothing needs a gradient; what looks into
    calls (forward-mode differentiation, transforms, the tracer) still meets ``apply``."""
    x = torch.ones(3, requires_grad=True)
    y = call(_Double, x)
    assert y.requires_grad and _Double.last == (True,)
    (g,) = torch.autograd.grad(y.sum(), x)
    assert torch.equal(g, torch.full((3,), 2.0))
    with torch.no_grad():
        y = call(_Double, x)
        assert not y.requires_grad and not any(_Double.last) and torch.equal(y, torch.full((3,), 2.0))
        with forward_ad.dual_level(), pytest.raises(Exception):
            call(_Double, forward_ad.make_dual(x.detach(), torch.ones(3)))
        with pytest.raises(Exception):
            torch.func.vmap(lambda t: call(_Double, t))(torch.ones(2, 3))
        traced = torch.jit.trace(lambda t: call(_Double, t), (torch.ones(3),), check_trace=False)
        assert "PythonOp" in str(traced.graph) or "_Double" in str(traced.graph)
    with torch.inference_mode():
        assert torch.equal(call(_Double, torch.ones(3)), torch.full((3,), 2.0))


class _Address(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x):
        return torch.tensor(x.data_ptr())

    @staticmethod
    def backward(ctx, g):
        return None


def test_call_on_a_tensor_that_outlived_its_transform():
    kept = []
    torch.func.grad(lambda t: (kept.append(t), (t * t).sum())[1])(torch.ones(3))
    with torch.no_grad():
        assert call(_Address, kept[0]).item() == _Address.apply(kept[0]).item() != 0


def test_kernels_let_their_successor_in_after_their_tensor_memory():
    """A successor that starts early must not take tensor memory that the kernel in front has yet to allocate, since it waits
    for that kernel: grid_go() follows the allocation in the warp that allocates."""
    import re

    found = 0
    for src in build.sources():
        code = re.sub(r"//[^\n]*", "", src.read_text())
        for kernel in code.split("__global__")[1:]:
            if "tmem_alloc<" not in kernel or "grid_go(" not in kernel:
                continue
            found += 1
            alloc, go = kernel.index("tmem_alloc<"), kernel.index("grid_go(")
            # one block of one warp: nothing between the two closes it
            assert alloc < go and "}" not in kernel[alloc:go], src.name
    assert found == 4
