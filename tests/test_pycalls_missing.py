"""A tree whose call module is not there: the binding makes the same calls
through ctypes, and the build leaves the module out instead of failing."""
from __future__ import annotations

import os
import subprocess
import sys
import sysconfig

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = """
import sys
if sys.argv[1] == "without":
    sys.modules["barbu_gb300._hscalls"] = None  # import raises ImportError
import numpy as np
from barbu_gb300 import hairsim
hairsim.lib()
assert (hairsim._calls is hairsim._CtypesCalls) == (sys.argv[1] == "without")
g = object.__new__(hairsim.Groom)
g.h = None  # the library refuses a null groom
for call in (lambda: g.set_wind(np.zeros(3, np.float32)), lambda: g.set_spheres(np.zeros((2, 4))),
             lambda: g.set_bounding_sphere([0, 0, 0, 1]), lambda: g.set_root_transform(np.eye(4)),
             lambda: g.set_bone_matrices(np.zeros((1, 16), np.float32)), lambda: g.update(1 / 60),
             lambda: g.set_wind(np.zeros(4, np.float32)), lambda: g.update("x")):
    try:
        call()
        print("no error")
    except Exception as e:
        print(type(e).__name__, e)
"""


def run(mode):
    r = subprocess.run([sys.executable, "-c", PROGRAM, mode], capture_output=True, text=True, cwd=ROOT)
    assert r.returncode == 0, r.stderr
    return r.stdout.splitlines()


def test_same_calls_without_the_module(built_library):
    from barbu_gb300 import build
    without = run("without")
    assert len(without) == 8 and all(line.startswith("HairSimError") for line in without[:6])
    assert without[6].startswith("ValueError") and "ArgumentError" in without[7]
    if os.path.exists(build.CALLS) or build.build_calls():
        assert run("with") == without


def test_build_without_python_headers(tmp_path, monkeypatch, capsys):
    from barbu_gb300 import build
    old = tmp_path / "_hscalls.so"
    old.write_bytes(b"of older sources")
    monkeypatch.setattr(build, "CALLS", str(old))
    monkeypatch.setattr(build.sysconfig, "get_paths", lambda *a: {"include": str(tmp_path)})
    assert build.build_calls() is None
    assert "ctypes" in capsys.readouterr().err and not old.exists()


def test_build_without_a_compiler(tmp_path, monkeypatch, capsys):
    from barbu_gb300 import build
    monkeypatch.setattr(build, "CALLS", str(tmp_path / "_hscalls.so"))
    monkeypatch.setattr(build.shutil, "which", lambda name: None)
    monkeypatch.setenv("PATH", str(tmp_path))
    assert build.build_calls() is None
    assert "ctypes" in capsys.readouterr().err


def test_module_carries_the_interpreters_tag():
    from barbu_gb300 import build
    assert build.CALLS.endswith(sysconfig.get_config_var("EXT_SUFFIX"))
