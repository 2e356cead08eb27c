"""The extension that calls the launchers (csrc/host_call.cpp): what it takes for a parameter, what it refuses, and that every parameter
arrives where the launcher looks for it - integers beyond the registers, floats between them, whole 64-bit numbers."""
import ctypes
import os
import subprocess
import sys

import pytest
import torch

SOURCE = r"""
#include <stdint.h>
#include <string.h>
static int64_t seen[64]; static float floats[8];
extern "C" int many(int a, void* b, float f0, int c, long long d, void* e, int g, float f1, int h, int i, void* j, float f2, int k, long long l,
                    int m, int n, void* o, int p, int q, int r) {
    const int64_t all[] = {a, (int64_t)b, c, d, (int64_t)e, g, h, i, (int64_t)j, k, l, m, n, (int64_t)o, p, q, r};
    memcpy(seen, all, sizeof(all)); floats[0] = f0; floats[1] = f1; floats[2] = f2;
    return a - 3;
}
extern "C" int64_t look(int i) { return seen[i]; }
extern "C" float look_float(int i) { return floats[i]; }
"""


@pytest.fixture(scope="module")
def calls():
    from kvcache_b200.kernels import api
    return api._host_calls()


@pytest.fixture(scope="module")
def library(tmp_path_factory):
    folder = tmp_path_factory.mktemp("calls")
    (folder / "many.cpp").write_text(SOURCE)
    subprocess.run(["g++", "-O1", "-shared", "-fPIC", "-o", folder / "many.so", folder / "many.cpp"], check=True)
    return ctypes.CDLL(str(folder / "many.so"))


def test_every_parameter_arrives(calls, library):
    many = calls.Call(ctypes.cast(library.many, ctypes.c_void_p).value, "ipfilpifiipfiliipiii", "many")
    args = [-7, 1 << 47, 0.25, True, -(1 << 60), None, 5, -1.5, 6, 7, ctypes.c_void_p(99), 3, 8, 1 << 40, 9, 10, ctypes.c_void_p(0), -11, 12, -(1 << 31)]
    assert many(*args) == -10
    library.look.restype, library.look_float.restype = ctypes.c_int64, ctypes.c_float
    want = [-7, 1 << 47, 1, -(1 << 60), 0, 5, 6, 7, 99, 8, 1 << 40, 9, 10, 0, -11, 12, -(1 << 31)]
    assert [library.look(i) for i in range(len(want))] == want
    assert [library.look_float(i) for i in range(3)] == [0.25, -1.5, 3.0]
    with pytest.raises(TypeError):
        many(*args[:-1])
    for place, wrong, error in ((0, 1 << 31, OverflowError), (0, 1.5, TypeError), (2, "x", TypeError), (1, 1.5, (TypeError, AttributeError)), (4, 1 << 64, OverflowError)):
        with pytest.raises(error):
            many(*args[:place], wrong, *args[place + 1:])


def test_parameters_that_may_be_left_out(calls, library):
    many = calls.Call(ctypes.cast(library.many, ctypes.c_void_p).value, "ipfilpifiipfiliip|iii", "many")
    args = [4, None, 0.5, 1, 2, None, 5, 1.5, 6, 7, None, 3.0, 8, 9, 10, 11, ctypes.c_void_p(12), 13, 14, 15]
    library.look.restype = ctypes.c_int64
    for given in (20, 18, 17):
        assert many(*args[:given]) == 1
        assert [library.look(i) for i in (13, 14, 15, 16)] == [12] + [v if 17 + i < given else 0 for i, v in enumerate((13, 14, 15))]
    for wrong in (args[:16], args + [1]):
        with pytest.raises(TypeError):
            many(*wrong)


def test_tensors_that_a_launcher_cannot_take(calls, library):
    from kvcache_b200.kernels.api import KernelError, _ptr
    many = calls.Call(ctypes.cast(library.many, ctypes.c_void_p).value, "ipfilpifiipfiliipiii", "many")
    args = [1, None, 0.0, 1, 1, None, 1, 0.0, 1, 1, None, 0.0, 1, 1, 1, 1, None, 1, 1, 1]
    assert _ptr(None) == 0
    for t in (torch.zeros(4), torch.zeros(4, 4).t()[:, 1:]):
        with pytest.raises(KernelError):
            _ptr(t)
        with pytest.raises(KernelError):
            many(args[0], t, *args[2:])
    with pytest.raises(ValueError):
        calls.Call(1, "p" * 41, "too many")
    with pytest.raises(ValueError):
        calls.Call(1, "x", "unknown")


class _AnswersInPython(torch.Tensor):
    """A tensor whose questions are answered in Python, by an exception."""
    @staticmethod
    def __new__(cls):
        return torch.Tensor._make_wrapper_subclass(cls, (4,), dispatch_sizes_strides_policy="strides")

    @classmethod
    def __torch_dispatch__(cls, func, types, args=(), kwargs=None):
        raise ValueError("not to be asked")


QUESTIONS = """
import torch, warnings
warnings.simplefilter("ignore")
from kvcache_b200.kernels import api
from test_host_call import _AnswersInPython
call = api._host_calls().Call(1, "p", "never called")
for make, error in ((lambda: torch.eye(4).to_sparse_csr(), RuntimeError), (_AnswersInPython, ValueError)):
    for ask in (api._ptr, call):
        try:
            ask(make())
        except error:
            print("raised")
"""


def test_tensors_whose_questions_throw():
    """An exception in Python for each, not the end of the process (a child, since an exception that leaves C code ends it)."""
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    done = subprocess.run([sys.executable, "-c", QUESTIONS], capture_output=True, text=True,
                          env=dict(os.environ, PYTHONPATH=os.pathsep.join([root, os.path.dirname(os.path.abspath(__file__))])))
    assert done.returncode == 0 and done.stdout.split() == ["raised"] * 4, done.stderr[-500:]


def test_a_missing_header_is_named(monkeypatch, tmp_path):
    import sysconfig
    from kvcache_b200.kernels import build
    paths = dict(sysconfig.get_paths(), include=str(tmp_path))
    monkeypatch.setattr(sysconfig, "get_paths", lambda: paths)
    with pytest.raises(build.BuildError, match="Python.h"):
        build.compile_module("host_call", force=True)
