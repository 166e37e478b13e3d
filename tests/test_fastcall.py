"""The Python binding's calls through the C extension (axhel_b200/pyext/fastcall.c):
they take and refuse what the C-ABI's declared argument types do, as ctypes
does.  No GPU: every call ends at an argument check or is a no-op (n = 0)."""
import ctypes as C
import os
import subprocess
import sys

import numpy as np
import pytest

from axhel_b200 import capi

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def fake(address=64):
    """An NTT whose handle is never read: the calls below are refused before."""
    t = capi.NTT.__new__(capi.NTT)
    t.h = C.c_void_p(address)
    t.close = lambda: None  # __del__ must not release it
    return t


# An integer is not None or a sequence, an address is not a sequence.
@pytest.mark.parametrize("call", [
    "capi.mul(0, 0, 0, None, 17, 1)",
    "capi.mul(8, 8, 8, 0, [17], 1)",
    "capi.mul(8, 8, 8, (0,), 17, 1)",
    "capi.add([0], 0, 0, 0, 97)",
    "capi.add(0, (1, 2), 0, 0, 97)",
    "capi.add(0, 0, None, 0, 97, scalar=True)",
    "capi.fma(0, 0, None, 0, 0, 97, 1)",
    "capi.reduce(0, 0, 0, None, 4, 1)",
    "capi.add(0, 0, 0, 0.0, 97)",
    "capi.add(0, 0, 0, 0, 97, stream=[0])",
    "capi.tensor_product(0, 0, 0, 0, 0, 0, 0, None, 0, [97])",
    "capi.forward_batch([], 8, 8, None)",
    "capi.product_batch([], 8, [8], 8, 1)",
])
def test_arguments_of_another_type_are_refused(call):
    with pytest.raises(C.ArgumentError):
        eval(call)


# A list of handles holds NTT objects, nothing else.  (In a process of its
# own: an address taken for a handle would be read.)
@pytest.mark.parametrize("ntts", ["[64]", "[None]", "(64, 128)", "['x']", "[object()]"])
def test_handles_are_ntt_objects(ntts):
    code = ("from axhel_b200 import capi\n"
            f"try: capi.forward_batch({ntts}, 8, 8, 1)\n"
            "except AttributeError: print('refused')\n")
    r = subprocess.run([sys.executable, "-c", code], cwd=ROOT, capture_output=True, text=True)
    assert (r.returncode, r.stdout) == (0, "refused\n"), r.stderr


@pytest.mark.parametrize("call", ["capi.forward_batch((t for t in [fake()]), 8, 8, 0)",
                                  "capi.tensor_product(0, 0, 0, 0, 0, 0, 0, 0, 0, (q for q in [97]))"])
def test_sequences_without_a_length_are_refused(call):
    with pytest.raises(TypeError):
        eval(call)


def test_kinds_are_the_declared_types():
    kind = {C.c_uint64: "i", C.c_void_p: "p", C.POINTER(C.c_void_p): "h"}
    for name, kinds in capi._HOT.items():
        declared = getattr(capi.lib(), "axhel_cuda_" + name).argtypes
        assert kinds.replace("a", "p") == "".join(kind[t] for t in declared), name


def test_integers_and_addresses_are_taken():
    capi.add(None, None, None, 0, 97, stream=None)          # no data
    capi.add(0, 0, 0, np.uint64(0), np.int64(97))           # integers with __index__
    capi.add(C.c_void_p(0), 0, 0, 0, 97, C.c_void_p(0))     # addresses as ctypes objects
    capi.tensor_product(0, 0, 0, 0, 0, 0, 0, 0, 0, np.array([97, 101], np.uint64))


@pytest.mark.parametrize("count,status", [(0, 1), (65, 4), (300, 4)])
def test_handle_lists_of_any_length(count, status):
    """None, one more than a batch takes, and more than the extension's own array holds."""
    for ntts in ([fake()] * count, (fake(),) * count):
        with pytest.raises(capi.AxhelError) as e:
            capi.forward_batch(ntts, 8, 8, 1)
        assert e.value.status == status
        with pytest.raises(capi.AxhelError) as e:
            capi.chain_fma_batch(ntts, 8, 8, [1] * count, 0, 1)
        assert e.value.status == status


def test_closed_handle_is_refused():
    t = fake(0)
    for call in (lambda: t.forward(8, 8), lambda: t.inverse(8, 8), lambda: capi.forward_batch([t], 8, 8, 1)):
        with pytest.raises(capi.AxhelError) as e:
            call()
        assert e.value.status == 1


def test_replaced_handle_is_the_one_passed():
    """In a process of its own: a handle kept from before would be read."""
    code = ("import ctypes as C\n"
            "from axhel_b200 import capi\n"
            "t = capi.NTT(8, 17, handle=C.c_void_p(64))\n"
            "t.h = C.c_void_p(0)\n"
            "for call in (lambda: t.forward(8, 8), lambda: capi.forward_batch([t], 8, 8, 1)):\n"
            "    try: call()\n"
            "    except capi.AxhelError as e: print(e.status)\n")
    r = subprocess.run([sys.executable, "-c", code], cwd=ROOT, capture_output=True, text=True)
    assert (r.returncode, r.stdout) == (0, "1\n1\n"), r.stderr


WITHOUT = "import sys\nsys.modules['axhel_b200._fastcall'] = None\n"


def test_calls_without_the_extension():
    code = WITHOUT + ("from axhel_b200 import capi\n"
                      "capi.add(0, 0, 0, 0, 97)\n"
                      "capi.tensor_product(0, 0, 0, 0, 0, 0, 0, 0, 0, [97])\n"
                      "try: capi.forward_batch([], 8, 8, 1)\n"
                      "except capi.AxhelError as e: print(e.status)\n"
                      "try: capi.mul(0, 0, 0, None, 17, 1)\n"
                      "except capi.C.ArgumentError: print('refused')\n")
    r = subprocess.run([sys.executable, "-c", code], cwd=ROOT, capture_output=True, text=True)
    assert (r.returncode, r.stdout) == (0, "1\nrefused\n"), r.stderr


@pytest.mark.parametrize("missing", ["headers", "compiler"])
def test_build_without_python_headers_or_compiler(tmp_path, monkeypatch, capsys, missing):
    """The library builds for C and C++ callers; Python's go through ctypes."""
    from axhel_b200 import build

    (tmp_path / "pyext").mkdir()
    (tmp_path / "pyext" / "fastcall.c").write_text("#include <Python.h>\n")
    monkeypatch.setattr(build, "PKG", str(tmp_path))
    if missing == "headers":
        import sysconfig

        monkeypatch.setattr(sysconfig, "get_paths", lambda: {"include": str(tmp_path)})
    else:
        monkeypatch.setenv("PATH", str(tmp_path))
    build.build_pyext()
    assert not (tmp_path / "_fastcall.so").exists()
    assert "_fastcall" in capsys.readouterr().err
