"""The library linked with a stand-in for the CUDA runtime (fake_cudart.cpp), for tests of its host
code without a GPU: kernels and copies do nothing, but launches and limits are checked."""
import json
import os
import subprocess
import sys

import pytest

from helpers import ROOT

PKG = os.path.join(ROOT, "heavy-disks_b200")
HEAD = """import sys
sys.path.insert(0, sys.argv[1])
import diskgpu as D
D.LIB_PATH, arg = sys.argv[2:]
"""


@pytest.fixture(scope="session")
def fake_lib(tmp_path_factory):
    subprocess.run(["make", "-s", "-C", PKG], check=True)
    out = str(tmp_path_factory.mktemp("fake") / "libdiskgpu_fake.so")
    objs = [os.path.join(PKG, "build", f) for f in sorted(os.listdir(os.path.join(PKG, "build"))) if f.endswith(".o")]
    inc = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")
    subprocess.run(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", "-I" + inc,
                    os.path.join(ROOT, "tests", "fake_cudart.cpp"), *objs, "-o", out], check=True)
    return out


def fake_child(lib, code, arg):
    """The last line that `code` prints, as JSON; it finds the binding as D and `arg` as JSON text."""
    r = subprocess.run([sys.executable, "-c", HEAD + code, PKG, lib, json.dumps(arg)], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-2000:]
    return json.loads(r.stdout.splitlines()[-1])
