"""The per-matrix calls of the Python binding: the module that passes their arguments is tied to no interpreter, and without it the same calls go
through ctypes, with the same results.  No GPU: a null context is refused by the library itself."""
import subprocess
import sys
from pathlib import Path

import numpy as np
import pytest

ROOT = Path(__file__).resolve().parent.parent


def routes(pkg, monkeypatch, tmp_path):
    yield "module", pkg._load_fastcall()
    other = tmp_path / "other.so"
    other.write_bytes(b"a module of another interpreter")
    for path in (tmp_path / "missing.so", other):                                     # not built; not loadable
        monkeypatch.setattr(pkg, "_fast", None)
        monkeypatch.setattr(pkg, "FAST_PATH", path)
        yield path.name, pkg._load_fastcall()


def test_every_route_makes_the_same_calls(pkg, monkeypatch, tmp_path):
    x, xq, xd, y = np.zeros(64, np.float32), np.zeros(64, np.int8), np.zeros(2, np.float16), np.zeros(32, np.float32)
    seen = []
    for name, f in routes(pkg, monkeypatch, tmp_path):
        seen.append(type(f).__name__)
        assert f.quant_q8(None, x, xq, xd, None, 1) == 1, name                          # MI_ERR_INVALID
        assert f.quant_q8(None, x.ctypes.data, xq, xd, 64, 1) == 1, name
        assert f.gemv_q4_q8(None, None, xq, xd, None, y, 0, 0) == 1, name
        assert f.gemm_q4_q8(None, None, xq, xd, 2, None, y) == 1, name
        with pytest.raises((TypeError, AttributeError)):
            f.gemv_q4_q8(None, None, "not a tensor", xd, None, y, 0, 0)
        with pytest.raises(TypeError):
            f.gemv_q4_q8(None, None, xq)
    assert seen[1:] == ["_CtypesCalls", "_CtypesCalls"]


def test_the_module_uses_the_limited_api_only(pkg):
    if not pkg.FAST_PATH.exists():
        pytest.skip("not built")
    names = subprocess.run(["nm", "-D", "--undefined-only", str(pkg.FAST_PATH)], capture_output=True, text=True, check=True).stdout.split()
    private = [n for n in names if n.startswith("_Py") and n not in ("_Py_NoneStruct", "_Py_Dealloc")]        # those two are part of it
    assert not private, private
    assert "Py_LIMITED_API 0x030A0000" in (ROOT / "nano-inference_b200" / "host" / "fastcall.cpp").read_text()


def test_a_missing_library_is_still_an_error(pkg):
    code = ("import importlib.util, sys; s = importlib.util.spec_from_file_location('nano_inference_b200', sys.argv[1]); m = importlib.util.module_from_spec(s);"
            "s.loader.exec_module(m); m.LIB_PATH = m.LIB_PATH.parent / 'missing.so'; m._load_fastcall()")
    r = subprocess.run([sys.executable, "-c", code, str(ROOT / "nano-inference_b200" / "__init__.py")], capture_output=True, text=True)
    assert r.returncode != 0 and "FileNotFoundError" in r.stderr
