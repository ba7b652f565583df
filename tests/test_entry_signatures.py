"""The argument types that the core library's entries are called with are those of their declarations: an argument too many would go
by ctypes' own rules, a pointer or stream as 32 bits."""
import ctypes
import os
import re

import pytest

from tensorline_b200 import ops

KINDS = {"int": ctypes.c_int, "float": ctypes.c_float, "long long": ctypes.c_longlong, "double": ctypes.c_double, "size_t": ctypes.c_size_t,
         "unsigned": ctypes.c_uint, "unsigned long long": ctypes.c_ulonglong, "cudaStream_t": ctypes.c_void_p}


def declared():
    found = {}
    folder = os.path.join(os.path.dirname(ops.__file__), "csrc")
    for source in ops.CORE_SOURCES:
        with open(os.path.join(folder, source)) as f:
            text = re.sub(r"//[^\n]*", "", f.read())
        for name, arguments in re.findall(r"TL_EXPORT\s+int\s+(\w+)\s*\(([^)]*)\)\s*\{", text):
            found[name] = []
            for a in filter(None, (x.strip() for x in arguments.split(","))):
                kind = re.sub(r"\bconst\b", "", a.rsplit(None, 1)[0] if "*" not in a else "*").strip()
                found[name].append(ctypes.c_void_p if kind == "*" else KINDS[kind])
    return found


@pytest.mark.parametrize("name", sorted(ops._SIGNATURES))
def test_arguments_as_declared(name):
    assert list(ops._SIGNATURES[name]) == declared()[name]
