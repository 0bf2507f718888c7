"""The ahead-of-time builds: when a library is made again."""

import os
import sys

import pytest
import torch

from tandem_b200.utils import build


@pytest.fixture
def commands(monkeypatch, tmp_path):
    """No compiler is run: what would be is taken down, and its output file holds the words that it was given."""
    lib, ran = str(tmp_path / "_ops.so"), []

    def run(cmd, verbose):
        ran.append(cmd)
        with open(cmd[cmd.index("-o") + 1], "w") as f:
            f.write("\n".join(cmd))

    monkeypatch.setattr(build, "OPS_LIB", lib)
    monkeypatch.setattr(build, "_run", run)
    monkeypatch.setattr(build, "nvcc_path", lambda: "/usr/local/cuda/bin/nvcc")
    if torch.version.cuda is None:
        monkeypatch.setattr(torch.version, "cuda", "12.8")
    return ran


def test_native_operators_are_built_again_for_another_torch(commands, monkeypatch):
    assert build.build_ops() == build.OPS_LIB and len(commands) == 1
    assert build.build_ops() == build.OPS_LIB and len(commands) == 1
    os.utime(build.OPS_LIB, (2e9, 2e9))  # however new it is
    monkeypatch.setattr(torch.version, "git_version", "0" * 40)
    assert build.build_ops() == build.OPS_LIB and len(commands) == 2
    assert build.build_ops() == build.OPS_LIB and len(commands) == 2


def test_the_built_library_names_what_it_was_built_for():
    if not os.path.exists(build.OPS_LIB):
        pytest.skip("not built")
    with open(build.OPS_LIB, "rb") as f:
        assert build.ops_built_for().encode() in f.read()


def test_build_beside_a_cpu_torch(monkeypatch):
    """The entry point builds what there is to build."""
    sys.path.insert(0, os.path.dirname(os.path.dirname(os.path.abspath(__file__))))
    import __graft_entry__ as entry

    if not os.path.exists(build.CUDA_LIB):
        pytest.skip("not built")
    monkeypatch.setattr(torch.version, "cuda", None)
    entry.build()


def test_ctypes_signatures_are_the_headers():
    """Every entry point that the Python operators call has the argument and result types of cuda/operators.h."""
    import ctypes
    import re

    from tandem_b200.ops import _lib, attention
    from tandem_b200.parallel.symm import cuda_lib

    if not os.path.exists(build.CUDA_LIB):
        pytest.skip("not built")
    with open(build.OPS_HEADER) as f:
        text = re.sub(r"//[^\n]*", "", f.read())
    plain = {"int": ctypes.c_int, "unsigned": ctypes.c_uint, "long long": ctypes.c_longlong, "float": ctypes.c_float, "void": None}
    pointers = {ctypes.c_void_p, ctypes.c_char_p, ctypes.POINTER(ctypes.c_int), ctypes.POINTER(ctypes.c_longlong), ctypes.POINTER(ctypes.c_void_p)}

    def kind(declared):
        declared = declared.strip()
        return "pointer" if "*" in declared or declared.startswith("cudaStream_t") else plain[declared]

    _lib.lib(), attention._fns()
    declarations = re.findall(r"^([a-z][\w* ]*?)\b(tb_\w+)\(([^)]*)\);", text, re.M)
    assert len(declarations) == 26
    for result, name, arguments in declarations:
        fn = getattr(cuda_lib(), name)
        given = [re.sub(r"\w+$", "", a.strip()) if "*" not in a else a for a in arguments.split(",") if a.strip()]
        want = [kind(a) for a in given]
        got = ["pointer" if t in pointers else t for t in (fn.argtypes or [])]
        assert got == want, name
        assert ("pointer" if fn.restype in pointers else fn.restype) == kind(result), name
