"""The ctypes mirrors of the header's structs have the header's fields, in its order, at
its offsets: a field added on one side alone would move every pointer after it."""

import ctypes
import re
from pathlib import Path

import pytest

from matvis_b200 import _lib

HEADER = Path(__file__).resolve().parents[1] / "include" / "matvis_b200.h"
SCALARS = {"int": ctypes.c_int, "int64_t": ctypes.c_int64, "size_t": ctypes.c_size_t, "float": ctypes.c_float,
           "double": ctypes.c_double, "int32_t": ctypes.c_int32}


def _header_struct(name):
    """A ctypes structure laid out from the header's declaration (natural C alignment)."""
    text = re.sub(r"/\*.*?\*/", "", HEADER.read_text(), flags=re.S)
    (body,) = re.findall(r"typedef struct \{([^}]*)\} %s;" % name, text)
    fields = []
    for decl in filter(None, (d.strip() for d in body.split(";"))):
        decl = decl.replace("const", " ")
        base, rest = re.match(r"\s*(\w+)(.*)", decl, re.S).groups()
        for item in rest.split(","):
            pointer = "*" in item
            fields.append((item.replace("*", "").strip(), ctypes.c_void_p if pointer else SCALARS[base]))
    return type(name, (ctypes.Structure,), {"_fields_": fields})


@pytest.mark.parametrize("name,mirror", [("mvb_job", _lib.Job), ("mvb_herk_group", _lib.HerkGroup)])
def test_layout(name, mirror):
    want = _header_struct(name)
    layout = lambda s: [(n, getattr(s, n).offset, getattr(s, n).size) for n, _ in s._fields_]
    assert layout(mirror) == layout(want)
    assert ctypes.sizeof(mirror) == ctypes.sizeof(want)
    assert [t for _, t in mirror._fields_] == [t for _, t in want._fields_]


def test_job_size():
    """What a C compiler makes of the header (x86-64): both parsed and mirrored layouts could be wrong alike."""
    assert (ctypes.sizeof(_lib.Job), _lib.Job.out_c128.offset) == (424, 416)
