"""A checkout without built files builds through the entry point and runs what it built, in one process."""
import os
import re
import shutil
import subprocess
import sys
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent

# Stands for nvcc, which takes minutes: the library is a C file that defines every symbol the header declares.
FAKE_NVCC = """#!{python}
import subprocess, sys
out = sys.argv[sys.argv.index("-o") + 1]
if "-c" in sys.argv:
    open(out, "w").close()
else:
    subprocess.run(["gcc", "-shared", "-fPIC", "-w", "-o", out, {stub!r}], check=True)
"""


@pytest.fixture
def checkout(tmp_path):
    skip = shutil.ignore_patterns("*.so", "*.so.host", "build", "__pycache__")
    for part in ("nuvec_b200", "include", "oracle"):
        shutil.copytree(ROOT / part, tmp_path / part, ignore=skip)
    shutil.copy(ROOT / "__graft_entry__.py", tmp_path)
    stub = tmp_path / "stub.c"
    names = sorted(set(re.findall(r"\b(nvc_[a-z0-9_]+)\s*\(", (ROOT / "include" / "nuvec_cuda.h").read_text())))
    stub.write_text("".join(f"int {n}() {{ return 0; }}\n" for n in names))
    nvcc = tmp_path / "nvcc"
    nvcc.write_text(FAKE_NVCC.format(python=sys.executable, stub=str(stub)))
    nvcc.chmod(0o755)

    def run(code):
        env = dict(os.environ, NVCC=str(nvcc), PYTHONPATH="")
        return subprocess.run([sys.executable, "-c", code], cwd=tmp_path, env=env, capture_output=True, text=True)

    run.root = tmp_path
    return run


BUILD_AND_USE = """
import __graft_entry__ as entry
entry.build()
import nuvec_b200 as nv
from nuvec_b200 import _native
assert issubclass(nv.Array, _native.ArrayBase) and issubclass(nv.Device, _native.DeviceBase)
"""


def test_clean_checkout_builds_and_loads_in_one_process(checkout):
    done = checkout(BUILD_AND_USE)
    assert done.returncode == 0, done.stderr
    native = list((checkout.root / "nuvec_b200").glob("_native*.so"))
    assert len(native) == 1
    native[0].unlink()  # the host path alone is missing
    done = checkout(BUILD_AND_USE)
    assert done.returncode == 0, done.stderr


def test_unbuilt_package_says_what_is_missing_and_a_broken_module_why(checkout):
    done = checkout("import nuvec_b200 as nv\nnv.Device")
    assert done.returncode != 0 and "nuvec_b200._native is missing: build it" in done.stderr
    assert checkout(BUILD_AND_USE).returncode == 0
    next((checkout.root / "nuvec_b200").glob("_native*.so")).write_bytes(b"not an object")
    done = checkout("import nuvec_b200 as nv\nnv.Device")
    assert done.returncode != 0 and "is missing" not in done.stderr and "_native" in done.stderr


def test_rebuilding_under_a_loaded_module_is_an_error(checkout):
    assert checkout(BUILD_AND_USE).returncode == 0
    done = checkout("import nuvec_b200 as nv\nnv.Array\nfrom nuvec_b200 import build\nbuild.build(force=True)")
    assert done.returncode != 0 and "start a new one" in done.stderr


def test_public_names_are_those_of_the_operators():
    import nuvec_b200 as nv
    from nuvec_b200 import ops
    names = {}
    exec("from nuvec_b200 import *", names)
    assert set(ops.__all__) | {"BF16", "F16", "F32", "I32", "U8", "U32"} <= set(names) & set(dir(nv))
    assert nv.ops is ops and nv.quantize is ops.quantize
    with pytest.raises(AttributeError):
        nv.no_such_name
