"""Rays that a wide pass hands on to the binary one: the indices in the hand-over lists are
checked against the batch (on the CPU; the lists themselves never hold such an index in a test)."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_an_index_past_the_batch_is_flagged_and_left_out(tmp_path):
    exe = str(tmp_path / "handed_on")
    cuda = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")
    subprocess.run([os.environ.get("BZR_CXX", "g++"), "-std=c++17", "-O1", "-I", cuda, "-I",
                    os.path.join(ROOT, "blazert_b200", "csrc"),
                    os.path.join(ROOT, "tests", "emu", "handed_on.cpp"), "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout


def test_a_leaf_past_the_arrays_is_flagged_before_its_box_is_read(tmp_path):
    exe = str(tmp_path / "bad_leaf")
    cuda = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")
    csrc = os.path.join(ROOT, "blazert_b200", "csrc")
    subprocess.run([os.environ.get("BZR_CXX", "g++"), "-std=c++17", "-O1", "-g",
                    "-fsanitize=address", "-ffp-contract=off", "-I", cuda, "-I", csrc, "-pthread",
                    os.path.join(ROOT, "tests", "emu", "bad_leaf.cpp"),
                    os.path.join(csrc, "scene.cpp"), os.path.join(csrc, "scene_io.cpp"),
                    "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
