"""The build entry point stands apart from the tests, and an image with leaf records (what flatten
makes unless told otherwise) can be walked on the host, as a program that fills KindView with
its records does."""
import os
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_build_needs_nothing_under_tests(tmp_path):
    """build() in a tree without tests/ (the built files are up to date, so nothing compiles)."""
    for name in ("blazert_b200", "include", "oracle", "__graft_entry__.py"):
        os.symlink(os.path.join(ROOT, name), tmp_path / name)
    env = {k: v for k, v in os.environ.items() if k != "PYTHONPATH"}
    r = subprocess.run([sys.executable, "-c", "import __graft_entry__ as g; g.build()"],
                       cwd=tmp_path, env=env, capture_output=True, text=True, timeout=1200)
    assert r.returncode == 0, r.stderr[-2000:]


@pytest.fixture(scope="module")
def walk(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("records") / "walk")
    csrc = os.path.join(ROOT, "blazert_b200", "csrc")
    cuda = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")
    subprocess.run([os.environ.get("BZR_CXX", "g++"), "-std=c++17", "-O1", "-ffp-contract=off",
                    "-I", cuda, "-I", csrc, "-pthread",
                    os.path.join(ROOT, "tests", "emu", "records_walk.cpp"),
                    os.path.join(csrc, "scene.cpp"), os.path.join(csrc, "scene_io.cpp"),
                    "-o", out], check=True)
    return out


@pytest.mark.parametrize("kind", ["mesh", "spheres", "planes"])
@pytest.mark.parametrize("prims", [1, 7, 2000])
def test_walk_of_leaf_records_equals_the_binary_walk(walk, kind, prims):
    r = subprocess.run([walk, kind, str(prims)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
