"""Building and loading without what is optional, no GPU."""
import os
import subprocess
import sys

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def run(code, *args):
    return subprocess.run([sys.executable, "-c", code, *args], cwd=ROOT, capture_output=True, text=True, timeout=300)


def test_the_c_library_builds_without_torch():
    # a Rust or C user's build: nothing but nvcc is run, torch cannot be imported
    r = run("""
import runpy, subprocess, sys
sys.modules["torch"] = None
ran = []
class Done:
    returncode, stdout, stderr = 0, "", ""
subprocess.run = lambda cmd, **kw: ran.append(cmd) or Done
sys.argv = ["_build.py", "--force"]
runpy.run_path("combsengine_b200/_build.py", run_name="__main__")
assert len(ran) == 1 and "nvcc" in ran[0][0], ran
""")
    assert r.returncode == 0, r.stderr
    assert "libcombskv.so" in r.stdout and "ctypes" in r.stdout


def test_the_package_works_without_the_native_calls():
    # no file for this torch and Python: the same answers through ctypes
    r = run("""
from combsengine_b200 import KVArena, _build, _lib
_build.pycall_path = lambda: "/nonexistent/_pycall.so"
assert _lib.native() is None
a = KVArena(1, 4, 2, 64, 64, num_pages=4)
s = a.new_seq()
a.begin_step_host_only([s], [20])
assert s.popn(3) == 3 and s.seq_len() == 17
try:
    a.begin_step([s], [1])
except Exception as e:
    print(type(e).__name__)
""")
    assert r.returncode == 0, r.stderr


def test_the_native_calls_name_the_torch_and_python_they_are_built_for():
    import sysconfig

    import torch

    from combsengine_b200 import _build, _lib
    assert torch.__version__ in _build.pycall_path() and _build.pycall_path().endswith(sysconfig.get_config_var("EXT_SUFFIX"))
    assert _lib.native() is not None and _lib.native().__file__ == _build.pycall_path()
