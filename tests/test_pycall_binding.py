"""The compiled binding of the decode calls: used where this interpreter has one, done without where it has none."""
import ctypes as C
import os
import sys
import sysconfig

import pytest

import cwick_b200
from cwick_b200 import build, lib

FAST = ["cwk_mla_decode", "cwk_gqa_decode", "cwk_dsa_select", "cwk_gdn_scan"]


def test_this_interpreter_has_the_compiled_calls():
    build.build()
    L = lib.load()
    for name in FAST:
        assert type(lib.fast(L, name)).__name__ == "builtin_function_or_method"


@pytest.mark.parametrize("name", FAST)
def test_without_the_module_the_calls_go_through_ctypes(monkeypatch, name):
    L = lib.load()
    monkeypatch.delattr(cwick_b200, "_pycall", raising=False)
    monkeypatch.setitem(sys.modules, "cwick_b200._pycall", None)        # what an import finds that must fail
    fn = lib.fast(L, name)
    assert fn is getattr(L, name)
    args = [0.0 if a is C.c_float else None if a is C.c_void_p else 1 for a in lib.SIGNATURES[name][1]]
    assert fn(*args) == lib.ERR_ARGUMENT


def test_the_file_is_this_interpreters_own(monkeypatch, tmp_path):
    """Another interpreter looks for another name; an untagged file of an earlier build, which it would load, does not stay."""
    assert os.path.basename(build.PYCALL) == "_pycall" + sysconfig.get_config_var("EXT_SUFFIX")
    monkeypatch.setattr(build, "PYCALL", str(tmp_path / os.path.basename(build.PYCALL)))
    untagged = os.path.join(build.HERE, "_pycall.so")
    open(untagged, "w").close()
    build.build_pycall()
    assert os.path.exists(build.PYCALL) and not os.path.exists(untagged)
    before = os.path.getmtime(build.PYCALL)
    build.build_pycall()                                                # up to date: nothing to do
    assert os.path.getmtime(build.PYCALL) == before


def test_a_failed_build_of_the_module_is_no_failed_build(monkeypatch, tmp_path, capsys):
    monkeypatch.setattr(build, "PYCALL", str(tmp_path / "_pycall.so"))
    monkeypatch.setenv("CC", "false")
    build.build_pycall()
    assert "ctypes" in capsys.readouterr().err and not os.path.exists(build.PYCALL)
