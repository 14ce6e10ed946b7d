"""The FP64 mode walks the wide image (trace_core.cuh, RayD) and hands the rays that walk does not
cover to the binary walk.  Its results are the oracle's, as the binary walk's are: on rays that
it covers, that it hands on before they start (zero, tiny, huge and non-finite components, a
negative or NaN tmin) and that end their walk without a result (a hit that moves the hit distance
outward)."""
import numpy as np
import pytest

from blazert_b200 import workloads as W
from oracle.oracle import Oracle
from tests.emu.emu import EmuScene
from tests.helpers import mismatches, product_scene, to_numpy
from tests.scenes import axis_rays, edge_case_scenes, grid_mesh


def special_cases():
    rng = np.random.default_rng(41)
    out = [(name, spec, R.origins, R.directions, R.tmin, R.tmax)
           for name, spec, R in edge_case_scenes()]
    # a flat grid whose hits all lie at the boxes' own distance, rays through its edges and
    # vertices: hits of neighbouring triangles that differ by an ulp
    v, f = grid_mesh(33, 1.0 / 3.0)
    v = v @ W.rotation_to(np.array([[0.3, -0.5, 0.8]]) / np.sqrt(0.98))[0].T
    n = 20_000
    target = v[rng.integers(0, len(v), n)]
    target[n // 2:] = 0.5 * (target[n // 2:] + v[rng.integers(0, len(v), n - n // 2)])
    o = rng.uniform(-30.0, 30.0, (n, 3))
    out.append(("grid_vertices", W.SceneSpec().add_mesh(v, f), o, target - o, None, None))
    # spheres around and behind the origins: with tmin < 0 a hit behind the origin is reported
    # at its absolute distance, which can exceed the hit before it
    c, r = rng.uniform(-3.0, 3.0, (300, 3)), rng.uniform(0.1, 1.5, 300)
    o, d = rng.uniform(-3.0, 3.0, (n, 3)), rng.standard_normal((n, 3))
    tmin = rng.choice([0.0, -0.0, -4.0, -0.5, 1.0, np.nan], n)
    tmax = rng.choice([np.inf, 5.0, 2.0, 0.0, -1.0, np.nan], n)
    spheres = W.SceneSpec().add_spheres(c, r)
    out.append(("spheres_behind", spheres, o, d, tmin, None))
    out.append(("ranges", spheres, o, d, tmin, tmax))
    # concentric spheres a few ulps apart: norm(t d) of a closer one can round above the hit
    # before it, which moves the hit distance outward
    shells = W.SceneSpec().add_spheres(np.zeros((64, 3)) + 0.25,
                                       1.0 + rng.integers(-8, 9, 64) * 2.0 ** -52)
    so = 4.0 * rng.standard_normal((n, 3))
    out.append(("shells", shells, so, 0.25 + 0.4 * rng.standard_normal((n, 3)) - so, None, None))
    # components outside the covered range, and raw directions of every length
    d2 = d * 10.0 ** rng.uniform(-200.0, 200.0, (n, 1))
    d2[::7, 0] *= 1e-160
    d2[::11, 1] = 0.0
    d2[::13] = 0.0
    d2[::17, 2] = np.inf
    d2[::19, 0] = np.nan
    o2 = o.copy()
    o2[::23] *= 1e120
    out.append(("components", spheres, o2, d2, None, None))
    # planes and a mesh seen along the axes
    mix = W.mixed_primitives(n_rays=16, n_spheres=200, n_cylinders=20, n_planes=300, seed=12).scene
    mix.add_mesh(*W.icosphere(3))
    oa, da = axis_rays(rng, -100, 100, 4000)
    ob, db = rng.uniform(-120.0, 120.0, (8000, 3)), rng.standard_normal((8000, 3))
    out.append(("axis_and_random", mix, np.concatenate([oa, ob]), np.concatenate([da, db]), None,
                None))
    return out


CASES = special_cases()


@pytest.mark.parametrize("any_hit", [False, True], ids=["closest", "any"])
@pytest.mark.parametrize("case", CASES, ids=lambda c: c[0])
def test_wide_walk_equals_oracle(case, any_hit):
    _, spec, o, d, tmin, tmax = case
    with np.errstate(all="ignore"):
        ref = Oracle(spec).intersect(o, d, tmin, tmax, any_hit=any_hit)
        got = EmuScene(spec).intersect(o, d, tmin, tmax, mode="wide64", any_hit=any_hit)
    assert got["error_word"] == 0
    assert mismatches(got, ref) == []


@pytest.mark.gpu
@pytest.mark.parametrize("case", CASES, ids=lambda c: c[0])
def test_wide_kernels_equal_the_binary_kernels(case):
    """The default launch (wide walk, then the binary pass over the rays handed on) against the
    binary kernels, which the shared-memory stack selects."""
    import torch

    _, spec, o, d, tmin, tmax = case
    scene, binary = product_scene(spec), product_scene(spec)
    binary.tune(shared_stack=True)
    dev = lambda a: None if a is None else torch.from_numpy(np.ascontiguousarray(a)).cuda()
    args = [dev(np.tile(a, (40, 1)) if a is not None and a.ndim == 2 else
                (None if a is None else np.tile(a, 40))) for a in (o, d, tmin, tmax)]
    for any_hit in (False, True):
        ref = to_numpy(binary.intersectN(*args, any_hit=any_hit))
        for k in ("prim", "geom"):
            ref[k] = ref[k].view(np.uint32)
        assert mismatches(scene.intersectN(*args, any_hit=any_hit), ref) == []
    assert scene.check() == 0 and binary.check() == 0
    scene.close()
    binary.close()
