"""The native side of a launch against its Python twin: arguments of every kind in the order that a launcher declares them, in registers and
on the stack, and the checks' results and messages."""

import ctypes
import shutil
import subprocess

import pytest
import torch

from rusty_llama_b200.errors import KernelError
from rusty_llama_b200.kernels import build, host

SOURCE = """
#include <math.h>
#include <stddef.h>
static double seen[64];
double* last(void) { return seen; }
#define S(i, v) seen[i] = (double)(v)
int few(const void* a, int b, float c) { S(0, a == NULL); S(1, b); S(2, c); return -b; }
int none(void) { return -7; }
long long wide(int a) { return ((long long)a << 33) + 1; }
int many(const void* a, int b, float c, long long d, const void* e, int f, float g, int h, int i, unsigned j, int k, float l, long long m, int n,
         const void* o, float p, float q, int r, float s, int t, float u, const void* v) {
  S(0, a == NULL); S(1, b); S(2, c); S(3, d); S(4, e != NULL); S(5, f); S(6, g); S(7, h); S(8, i); S(9, j); S(10, k); S(11, l); S(12, m); S(13, n);
  S(14, o == NULL); S(15, p); S(16, q); S(17, r); S(18, s); S(19, t); S(20, u); S(21, (size_t)v & 0xffff);
  return r - t;
}
"""


def launchers():
    build.build_host_calls()
    native = build.load_host_calls(False)
    native.set_error(KernelError)
    return native, [native.launcher, host.PythonLauncher]


@pytest.fixture(scope="module")
def library(tmp_path_factory):
    if not shutil.which("gcc"):
        pytest.skip("no C compiler")
    d = tmp_path_factory.mktemp("host_calls")
    (d / "seen.c").write_text(SOURCE)
    subprocess.run(["gcc", "-O2", "-shared", "-fPIC", "-o", str(d / "seen.so"), str(d / "seen.c")], check=True)
    lib = ctypes.CDLL(str(d / "seen.so"))
    lib.last.restype = ctypes.POINTER(ctypes.c_double)
    return lib


def test_arguments_reach_the_launcher_as_declared(library):
    native, makers = launchers()
    at = lambda name: ctypes.cast(getattr(library, name), ctypes.c_void_p).value  # noqa: E731
    t = torch.zeros(8)
    args = (None, -3, 1.5, -(1 << 40), t, True, -2.25, 7, -8, 4000000000, 10, 0.5, 1 << 35, 13, None, 15.0, -16.0, 17, float("inf"), 19, 0.1, t)
    want = [1, -3, 1.5, -(1 << 40), 1, 1, -2.25, 7, -8, 4000000000, 10, 0.5, 1 << 35, 13, 1, 15, -16, 17, float("inf"), 19, ctypes.c_float(0.1).value, t.data_ptr() & 0xFFFF]
    for make in makers:
        assert make(at("few"), False)(t, 5, 2.5) == -5 and library.last()[:3] == [0.0, 5.0, 2.5]
        assert make(at("many"), False)(*args) == -2 and library.last()[:22] == want
        assert make(at("none"), False)() == -7 and make(at("wide"), True)(3) == (3 << 33) + 1
    few = native.launcher(at("few"), False)
    for wrong in (("x", 1, 1.0), (t, [1], 1.0), tuple([1.0] * 9), tuple([1] * 57)):
        with pytest.raises(TypeError):
            few(*wrong)
    with pytest.raises(RuntimeError):  # a C++ exception on the way is a Python one
        few(torch.sparse_coo_tensor(torch.tensor([[0]]), torch.tensor([1.0]), (2,)), 1, 1.0)


def test_checks_and_views_agree_with_python():
    native, _ = launchers()

    def outcome(f, *a, **k):
        try:
            return f(*a, **k)
        except KernelError as e:
            return str(e)

    t = torch.arange(24, dtype=torch.float32).view(4, 6)
    for a, k in (((1, "a"), {}), ((t, "b c"), {}), ((t, "b", torch.float32), {}), ((t.t(), "d"), dict(contiguous=False))):
        assert outcome(native.cuda, *a, **k) == outcome(host.python_cuda, *a, **k)
    for x in (t, t[:, 2:4], t.t(), t[0]):
        assert outcome(native.rows, x, "r") == outcome(host.python_rows, x, "r")
    assert torch.equal(native.columns(t, 1, 4), host.python_columns(t, 1, 4)) and native.columns(t, 1, 4).stride() == (6, 1)
    m = torch.zeros(3, 4, 2, 8)[:, :, 1]
    for x, y in ((m, None), (m, torch.zeros(3, 4, 2, 8)[:, :, 0]), (torch.zeros(8, 3, 4).transpose(0, 1), None)):
        assert native.matrices(x, y, m, "m") == host.python_matrices(x, y, m, "m")
    assert native.matrices(m, None, m, "m") == (3, 4, 8, 16, 64)
    e = native.empty(t, torch.bfloat16, 3, 5)
    assert e.dtype == torch.bfloat16 and tuple(e.shape) == (3, 5) and e.device == t.device
    w = torch.zeros(64, 64, dtype=torch.bfloat16)
    for x, y in ((w, w), (w[:, 1:], w), (w, w[:, 4:]), (w[:, :63], w), (w[:, 8:], w), (torch.zeros(4, 60, dtype=torch.bfloat16), w)):
        assert native.odd(x, y) == host.python_odd(x, y)


@pytest.mark.gpu
def test_the_native_side_is_what_launches():
    from rusty_llama_b200.kernels import ops

    assert host._module is not None and ops._cuda is host._module.cuda
    x = torch.zeros(4, 6, device="cuda")
    for a, k in (((x, "a", torch.bfloat16), {}), ((x.t(), "b"), {}), ((x, "c", torch.float32, True), {}), ((x.t(), "d"), dict(contiguous=False))):
        results = []
        for f in (host._module.cuda, host.python_cuda):
            try:
                results.append(f(*a, **k) is a[0])
            except KernelError as e:
                results.append(str(e))
        assert results[0] == results[1]
    assert host._module.stream() == host.python_stream()
    with torch.cuda.stream(torch.cuda.Stream()):
        assert host._module.stream() == host.python_stream() == torch.cuda.current_stream().cuda_stream
    with pytest.raises(torch.OutOfMemoryError):
        host._module.empty(x, torch.float32, 1 << 45)


def _exported():
    import os

    kinds = {}
    for name in build.source_names():
        with open(os.path.join(build.CSRC_DIR, name + ".cu")) as f:
            kinds.update(host.launcher_kinds(f.read()))
    return kinds


def test_arguments_of_another_kind_or_number_are_refused(library):
    """What ctypes refused stays refused: a float, None or a tensor of floats where a whole number goes moved every argument behind it."""
    native, makers = launchers()
    at = lambda name: ctypes.cast(getattr(library, name), ctypes.c_void_p).value  # noqa: E731
    t = torch.zeros(8)
    for make in makers:
        few = make(at("few"), False, "pif")
        assert few(t, torch.tensor(5), 2) == -5 and library.last()[:3] == [0.0, 5.0, 2.0]  # (whole numbers and floats of every sort, as ctypes took them)
        assert few(t.data_ptr(), True, torch.tensor(0.5)) == -1 and library.last()[:3] == [0.0, 1.0, 0.5]
        for wrong in ((t, 5.0, 2.0), (t, None, 2.0), (t, t, 2.0), (t, torch.tensor(1.0), 2.0), (t, 1, None), (t, 1, "x"), (t, 1, t), (1.0, 1, 1.0), ("x", 1, 1.0), (t, 1), (t, 1, 1.0, 1), ()):
            with pytest.raises((TypeError, RuntimeError, ValueError) if any(a is t for a in wrong[1:]) else TypeError):
                few(*wrong)
        with pytest.raises(TypeError):
            make(at("none"), False, "")(1)


def test_a_library_knows_what_its_launchers_take():
    if not shutil.which("nvcc"):
        pytest.skip("no CUDA compiler")
    takes = host.library("grouped_gemm").rl_grouped_gemm_takes
    assert takes(64, 8, 8) == 1
    for wrong in ((64.0, 8, 8), (64, None, 8), (64, 8), (64, 8, 8, 0)):
        with pytest.raises(TypeError):
            takes(*wrong)


def test_every_call_gives_a_launcher_as_many_arguments_as_it_takes():
    import ast
    import inspect

    from rusty_llama_b200.kernels import ops

    kinds, stars, seen = _exported(), {"_wt": 2, "_act": 2, "_bias_args": 2}, 0
    for call in ast.walk(ast.parse(inspect.getsource(ops))):
        if not (isinstance(call, ast.Call) and isinstance(call.func, ast.Attribute) and call.func.attr in kinds):
            continue
        n = 0
        for a in call.args:
            if not isinstance(a, ast.Starred):
                n += 1
            elif isinstance(a.value, ast.GeneratorExp):
                n += 3  # the three numbers of a pair of maps
            else:
                n += stars[a.value.func.id]
        assert n == len(kinds[call.func.attr][1]), call.func.attr
        seen += 1
    assert seen > 50


def test_importing_touches_neither_cuda_nor_a_compiler(tmp_path):
    import os
    import sys

    code = """
import os, subprocess, sys, torch
def never(*a, **k): raise AssertionError("called by the import")
torch.cuda.is_available = torch.cuda.device_count = torch.cuda.init = torch._C._cuda_getDeviceCount = subprocess.run = subprocess.Popen = never
import rusty_llama_b200
from rusty_llama_b200.kernels import host, linear, ops
assert (ops._cuda, linear._odd) == ((host.python_cuda, host.python_odd) if "_module" not in vars(host) else (host._module.cuda, host._module.odd))
assert ("_module" in vars(host)) == sys.argv[1].startswith("built")
"""
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    build.build_host_calls()
    subprocess.run([sys.executable, "-c", code, "built"], cwd=root, check=True)
    # where it is not built, in a folder of its own: Python until the first library
    empty = tmp_path / "empty"
    empty.mkdir()
    subprocess.run([sys.executable, "-c", code, "missing"], cwd=root, check=True, env=dict(os.environ, RUSTY_LLAMA_BUILD_DIR=str(empty)))
    assert not list(empty.iterdir())


def test_functions_are_native_from_the_first_library_on():
    if not shutil.which("nvcc"):
        pytest.skip("no CUDA compiler")
    from rusty_llama_b200.kernels import linear, ops

    build.build_host_calls()
    host.library("grouped_gemm")
    assert host._module is not None and ops._cuda is host._module.cuda and ops._empty is host.empty and linear._odd is host._module.odd


def test_one_process_builds_and_a_failure_is_remembered(tmp_path, monkeypatch):
    import os
    import threading

    monkeypatch.setattr(build, "_build_dir_cached", str(tmp_path))
    runs = tmp_path / "runs"
    tool = tmp_path / "compiler"
    tool.write_text(f"#!/bin/sh\necho run >> {runs}\nsleep 0.3\n[ -e {tmp_path}/works ] && echo built > $1\n")
    tool.chmod(0o755)
    monkeypatch.setattr(build, "_host_command", lambda out: [str(tool), out])
    with pytest.raises(KernelError):
        build.load_host_calls(True)
    assert build.load_host_calls(True) is None and build.load_host_calls(False) is None and len(runs.read_text().split()) == 1
    (tmp_path / "works").write_text("")
    several = [threading.Thread(target=build.build_host_calls) for _ in range(4)]
    for t in several:
        t.start()
    for t in several:
        t.join()
    assert len(runs.read_text().split()) == 2 and os.path.isfile(tmp_path / (build.HOST_CALLS + ".so"))
    flags = build._host_flags()
    before = build._host_fingerprint()
    monkeypatch.setattr(build, "_host_flags", lambda: flags + ["-O1"])
    assert build._host_fingerprint() != before


def test_refusals_agree_with_python(library):
    """What one side refuses the other does too, with the same kind of error and, where it is the library's own, the same words."""
    native, (make, python_make) = launchers()
    at = ctypes.cast(library.none, ctypes.c_void_p).value
    t, i, m = torch.zeros(4, 6), torch.zeros(()), torch.zeros(2, 2, 8)
    pairs = [
        (make(at, False), python_make(at, False), [tuple([1.0] * 9), tuple([1] * 57)]),
        (lambda k: make(at, False, k), lambda k: python_make(at, False, k), ["f" * 9, "i" * 57]),
        (make(at, False, "pif"), python_make(at, False, "pif"), [(t, 1), (1.5, 1, 1.0), (t, 1.5, 1.0), (t, 1, "x")]),
        (native.rows, host.python_rows, [(3, "r"), (t[0], "r"), (t.t(), "r")]),
        (native.matrices, host.python_matrices, [(t, None, m, "m"), (m.transpose(1, 2), None, m, "m"), (m, m[:1], m, "m"), (m, m.view(2, 8, 2).transpose(1, 2), m, "m"), (3, m, m, "m"),
                                                    (m, 3, m, "m"), (m, m, 3, "m"), (m, None, m.double(), "m"), (m, m.double(), m, "m")]),
        (native.odd, host.python_odd, [(t[0], t), (t.view(2, 2, 6), t), (t, i), (3, t), (t, 3)]),
        (native.empty, host.python_empty, [(t, torch.float32), (t, torch.float32, 1, 1, 1, 1, 1), (t, 3, 1), (3, torch.float32, 1), (t, torch.float32, -1)]),
        (native.columns, host.python_columns, [(t, 2, 9), (t, 7, 8), (t, 4, 2), (t[0], 0, 1), (3, 0, 1)]),
        (native.cuda, host.python_cuda, [(3, "a"), (t, "a")]),
    ]
    for one, other, calls in pairs:
        for args in calls:
            seen = []
            for f in (one, other):
                with pytest.raises(Exception) as e:
                    f(*(args if isinstance(args, tuple) else (args,)))
                words = str(e.value)
                seen.append((e.type, words if e.type is KernelError or "launcher" in words else ""))
            assert seen[0] == seen[1], (args, seen)
