"""Each kind's pass reads what the passes before it wrote (closest distances, the sort's order, the
zeroed counters) although its kernels overlap theirs: calls that follow each other on the same
buffers with other rays, several kinds, with and without the coherence sort, give the oracle's
results every time."""
import numpy as np
import pytest

from blazert_b200 import workloads as W
from oracle.oracle import Oracle
from tests.helpers import mismatches, product_scene, to_numpy

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sort", [False, True], ids=["plain", "sorted"])
@pytest.mark.parametrize("mode", ["fp64", "mixed"])
def test_repeated_calls_of_several_kinds(mode, sort):
    import torch

    n = 120_011  # above what the one launch of small batches takes, and above the sort's line
    spec = W.mixed_primitives(n_rays=1, n_spheres=600, n_cylinders=80, n_planes=60, seed=3).scene
    v, f = W.icosphere(4)
    mix = W.SceneSpec().add_mesh(50.0 * v, f)
    for k in spec.order:
        getattr(mix, "add_" + k)(*getattr(spec, k).values())
    scene, ora = product_scene(mix), Oracle(mix)
    scene.tune(sort=sort)
    rng = np.random.default_rng(17)
    sets = []
    for _ in range(3):
        o, d = rng.uniform(-120.0, 120.0, (n, 3)), rng.standard_normal((n, 3))
        d[::97] = [0.0, 0.0, -1.0]  # left out of the wide walks, scattered over the batch
        sets.append((torch.from_numpy(o).cuda(), torch.from_numpy(d).cuda(), ora.intersect(o, d)))
    o, d = torch.empty_like(sets[0][0]), torch.empty_like(sets[0][1])
    out = None
    for rep in range(30):
        so, sd, ref = sets[rep % 3]
        o.copy_(so)
        d.copy_(sd)
        out = scene.intersectN(o, d, mode=mode, out=out)
        got = to_numpy(out)
        for k in ("prim", "geom"):
            got[k] = got[k].view(np.uint32)
        assert mismatches(got, ref) == [], rep
    assert scene.check() == 0
    scene.close()


@pytest.mark.parametrize("mode", ["fp64", "mixed"])
@pytest.mark.parametrize("rays", ["axis", "mostly_axis", "far"])
def test_large_batches_the_wide_walk_hardly_covers(mode, rays):
    """Batches above the line from which a pass is left to the binary kernel as a whole when hardly
    any of its rays is covered: all axis-parallel, all but a few (the sample may or may not meet
    them), and far origins."""
    import torch

    n = 2_097_152 + 3_001 if mode == "fp64" and rays == "axis" else 800_003
    v, f = W.icosphere(4)
    mix = W.SceneSpec().add_mesh(v, f)
    mix.add_spheres(*W.mixed_primitives(n_rays=1, n_spheres=50, seed=3).scene.spheres.values())
    scene, ora = product_scene(mix), Oracle(mix)
    rng = np.random.default_rng(5)
    m = 50_021
    o, d = rng.uniform(-1.2, 1.2, (m, 3)), np.tile([0.0, 0.0, -1.0], (m, 1))
    o[:, 2] = 3.0
    if rays == "mostly_axis":
        d[::50] = rng.standard_normal((len(d[::50]), 3))
    if rays == "far":
        d[:] = rng.standard_normal((m, 3))
        o = rng.uniform(-1.2, 1.2, (m, 3)) - 3e18 * d
    ref = ora.intersect(o, d)
    idx = torch.arange(n, device="cuda") % m
    out = scene.intersectN(torch.from_numpy(o).cuda()[idx], torch.from_numpy(d).cuda()[idx],
                           mode=mode)
    idx = idx.cpu().numpy()
    got = to_numpy(out)
    for k in ("prim", "geom"):
        got[k] = got[k].view(np.uint32)
    assert mismatches(got, {k: ref[k][idx] for k in ("t", "uv", "normal", "prim", "geom",
                                                     "hit")}) == []
    assert scene.check() == 0
    scene.close()
