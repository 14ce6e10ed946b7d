"""Rays whose wide walk ends without a result are traced again by the binary walk.  Hits that exceed
the one before by rounding alone (coplanar triangles, concentric spheres, at a power of two as
well) do not end a walk: a batch of them must not be traced twice."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def redo_count(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("redo") / "redo_count")
    csrc = os.path.join(ROOT, "blazert_b200", "csrc")
    cuda = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")
    subprocess.run([os.environ.get("BZR_CXX", "g++"), "-std=c++17", "-O1", "-ffp-contract=off",
                    "-I", cuda, "-I", csrc, "-pthread",
                    os.path.join(ROOT, "tests", "emu", "redo_count.cpp"),
                    os.path.join(csrc, "scene.cpp"), os.path.join(csrc, "scene_io.cpp"),
                    "-o", out], check=True)
    return out


@pytest.mark.parametrize("case", ["coplanar", "floor", "shells", "tiny_negative_tmin"])
def test_rounding_does_not_end_a_walk(redo_count, case):
    r = subprocess.run([redo_count, case, "0"], capture_output=True, text=True)
    print(r.stdout)
    assert r.returncode == 0, r.stdout + r.stderr
