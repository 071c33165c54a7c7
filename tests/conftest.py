"""pytest configuration: the `gpu` marker, import path, and library fixtures."""
import json
import os
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(ROOT, "tim-vx_b200"))
sys.path.insert(0, ROOT)
sys.path.insert(0, os.path.join(ROOT, "tests"))


def pytest_configure(config):
    config.addinivalue_line("markers", "gpu: needs a CUDA device (run with -m gpu on a B200)")


def _ensure(path, make_dir):
    if not os.path.exists(path):
        subprocess.check_call(["make", "-C", make_dir], stdout=subprocess.DEVNULL)
    return path


@pytest.fixture(scope="session")
def oracle_lib():
    import oracle_paths
    _ensure(oracle_paths.ORACLE_LIB, os.path.join(ROOT, "oracle"))
    return oracle_paths.load(oracle_paths.ORACLE_LIB)


@pytest.fixture(scope="session")
def product_lib():
    """The CUDA library.  Missing library = hard failure, never a fallback."""
    import pyb2vx
    assert os.path.exists(pyb2vx.PRODUCT_LIB), "libb2vx.so is not built: run python -c 'import __graft_entry__ as g; g.build()'"
    return pyb2vx.load(pyb2vx.PRODUCT_LIB)


@pytest.fixture(scope="session")
def reference_cases():
    with open(os.path.join(ROOT, "tests", "golden", "reference_cases.json")) as f:
        return json.load(f)["cases"]


@pytest.fixture(scope="session")
def launch_rules(tmp_path_factory):
    """Asks the CUDA library's host-side launch rules through tests/cpp/launch_rules.cc (no GPU needed): questions as tuples of a name
    and whole numbers, answers as tuples."""
    import pyb2vx
    exe = str(tmp_path_factory.mktemp("rules") / "launch_rules")
    csrc = os.path.dirname(pyb2vx.PRODUCT_LIB)
    subprocess.check_call(["/usr/bin/g++", "-std=c++17", "-O1", "-Wall", "-Wextra", "-I" + csrc, "-I/usr/local/cuda/include",
                           os.path.join(ROOT, "tests", "cpp", "launch_rules.cc"), pyb2vx.PRODUCT_LIB, "-Wl,-rpath," + csrc, "-o", exe])

    def ask(questions):
        out = subprocess.run([exe] + [",".join(str(f) for f in q) for q in questions], capture_output=True, text=True, timeout=60)
        assert out.returncode == 0, out.stderr
        return [tuple(int(f) for f in line.split()) for line in out.stdout.splitlines()]
    return ask
