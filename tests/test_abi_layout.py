"""The structs that the ctypes mirror fills have the layout that a C compiler gives
include/gmk.h's, and the library exports nothing that the header does not declare."""
import ctypes
import os
import re
import shutil
import subprocess

import pytest

import gmkbe_b200 as G
from gmkbe_b200 import api
from conftest import ROOT

STRUCTS = {"gmk_opts": api._Opts, "gmk_stats": api._Stats, "gmk_task": api._Task, "gmk_collector": api._Collector}


@pytest.mark.parametrize("name", sorted(STRUCTS))
def test_struct_layouts_agree(tmp_path, name):
    cc = shutil.which("gcc") or shutil.which("cc")
    if cc is None:
        pytest.skip("no C compiler")
    fields = [f[0] for f in STRUCTS[name]._fields_]
    src = tmp_path / "l.c"
    src.write_text("#include \"gmk.h\"\n#include <stdio.h>\nint main(void) {\n"
                   + f"printf(\"%zu\\n\", sizeof({name}));\n"
                   + "".join(f"printf(\"%zu %zu\\n\", offsetof({name}, {f}), sizeof((({name}*)0)->{f}));\n"
                             for f in fields) + "return 0; }\n")
    exe = tmp_path / "l"
    subprocess.run([cc, "-I", os.path.join(ROOT, "include"), str(src), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True, check=True).stdout.split("\n")
    cls = STRUCTS[name]
    assert int(out[0]) == ctypes.sizeof(cls)
    for f, line in zip(fields, out[1:]):
        d = getattr(cls, f)
        assert (d.offset, d.size) == tuple(int(x) for x in line.split()), f


def test_every_exported_symbol_is_declared():
    text = open(os.path.join(ROOT, "include", "gmk.h")).read()
    declared = set(re.findall(r"\b(gmk_[a-z_]+)\s*\(", text)) - {"gmk_sink"}
    out = subprocess.run(["nm", "-D", "--defined-only", G.LIB_PATH], capture_output=True, text=True, check=True).stdout
    assert set(re.findall(r"\sT\s(gmk_\w+)", out)) == declared
