"""Rays whose raw direction is so long that the FP32 inverse of a component would be denormal: the
mixed mode's wide walk does not cover them (trace_core.cuh, RayW), and its results are the
oracle's for every length."""
import numpy as np
import pytest

from blazert_b200 import workloads as W
from oracle.oracle import Oracle
from tests.emu.emu import EmuScene
from tests.helpers import mismatches, product_scene, to_numpy


def _case(scale, seed):
    rng = np.random.default_rng(seed)
    n = 6000
    v, f = W.icosphere(3)
    spec = W.SceneSpec().add_mesh(scale * v, f)
    spec.add_spheres(scale * rng.uniform(-2.0, 2.0, (200, 3)), scale * rng.uniform(0.05, 0.3, 200))
    o = scale * rng.uniform(-3.0, 3.0, (n, 3))
    d = scale * rng.uniform(-2.0, 2.0, (n, 3)) - o
    d /= np.linalg.norm(d, axis=1)[:, None]
    # lengths about both ends of the covered range, and one component alone beyond it
    d *= 2.0 ** rng.choice([0, 95, 99, 100, 101, 126, 127, 130, 140, 148, 152, 200], (n, 1))
    d[::3] *= 2.0 ** rng.choice([0, 40], (len(d[::3]), 3))
    return spec, o, d


SCALES = [1.0, 1e9, 1e12, 1e15, 1e16]


@pytest.mark.parametrize("any_hit", [False, True], ids=["closest", "any"])
@pytest.mark.parametrize("scale", SCALES)
def test_long_directions_equal_oracle(scale, any_hit):
    for seed in range(4):
        spec, o, d = _case(scale, seed)
        ref = Oracle(spec).intersect(o, d, any_hit=any_hit)
        assert ref["hit"].any()
        got = EmuScene(spec).intersect(o, d, mode="mixed", any_hit=any_hit)
        assert got["error_word"] == 0
        assert mismatches(got, ref) == [], seed


@pytest.mark.gpu
@pytest.mark.parametrize("scale", SCALES)
def test_long_directions_on_the_gpu(scale):
    import torch

    spec, o, d = _case(scale, 9)
    scene, ref = product_scene(spec), Oracle(spec).intersect(o, d)
    reps = 12  # more rays than the one launch of small batches takes
    t = [torch.from_numpy(np.tile(a, (reps, 1))).cuda() for a in (o, d)]
    got = to_numpy(scene.intersectN(*t, mode="mixed"))
    want = {k: np.concatenate([ref[k]] * reps) for k in ("t", "uv", "normal", "prim", "geom", "hit")}
    for k in ("prim", "geom"):
        got[k] = got[k].view(np.uint32)
    assert mismatches(got, want) == []
    scene.close()
