"""The argument types that Python declares for the CUDA library's functions are those of their C declarations: a pointer passed as a 32-bit
number loses half of its bits, on some streams only."""
import ctypes
import importlib
import pathlib
import pkgutil
import re

import tunix_b200.ops
from tunix_b200 import _lib

_C = {"int": ctypes.c_int, "long long": ctypes.c_longlong, "float": ctypes.c_float, "unsigned long long": ctypes.c_ulonglong,
      "double": ctypes.c_double, "unsigned": ctypes.c_uint, "uint64_t": ctypes.c_uint64, "int64_t": ctypes.c_int64,
      "uint32_t": ctypes.c_uint32, "size_t": ctypes.c_size_t}


def _kind(param: str):
    param = " ".join(re.sub(r"\bconst\b|__restrict__", " ", param.split("=")[0]).split())
    if "*" in param or param.startswith("cudaStream_t") or param.endswith("]"):
        return "pointer"
    name = re.sub(r"\s*\w+$", "", param) or param
    return (ctypes.sizeof(_C[name]), name in ("float", "double")) if name in _C else None


def _declared(t):
    if t in (ctypes.c_void_p, ctypes.c_char_p) or hasattr(t, "contents"):
        return "pointer"
    return (ctypes.sizeof(t), t in (ctypes.c_float, ctypes.c_double))


def test_declared_argument_types_match_the_sources():
    for m in pkgutil.iter_modules(tunix_b200.ops.__path__):
        importlib.import_module("tunix_b200.ops." + m.name)
    found = {}
    for f in (pathlib.Path(_lib.__file__).parent / "csrc").glob("*.cu"):
        text = re.sub(r"//[^\n]*|/\*.*?\*/", "", f.read_text(), flags=re.S)
        for name, params in re.findall(r"TB_API\s+[\w\s\*]+?\b(tb_\w+)\s*\(([^)]*)\)\s*\{", text):
            found[name] = [_kind(p) for p in params.split(",")] if params.strip() not in ("", "void") else []
    sigs = _lib._CUDA_SIGS
    checked = 0
    for name, types in sigs.items():
        if name not in found or None in found[name]:
            continue
        assert [_declared(t) for t in types] == found[name], name
        checked += 1
    assert checked > 50
