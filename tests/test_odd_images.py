"""Rays that a wide pass leaves out, dealt to its first blocks in pieces: at sizes around their edges
(a run of 32, a piece of 8, the quarters of the batch) every ray is traced once, whether one, some or
most are left out."""
import numpy as np
import pytest

from blazert_b200 import workloads as W
from oracle.oracle import Oracle
from tests.helpers import mismatches, product_scene, to_numpy

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", ["fp64", "mixed"])
def test_left_out_rays_are_traced_once(mode):
    import torch

    v, f = W.icosphere(3)
    spec = W.SceneSpec().add_mesh(v, f)
    spec.add_spheres(*W.mixed_primitives(n_rays=1, n_spheres=40, seed=3).scene.spheres.values())
    scene, ora = product_scene(spec), Oracle(spec)
    rng = np.random.default_rng(12)
    m = 40_960 + 33
    o, d = rng.uniform(-1.5, 1.5, (m, 3)), rng.standard_normal((m, 3))
    o[:, 2] = 3.0
    d[:, 2] = -np.abs(d[:, 2]) - 1.0
    for n in (32_768, 32_769, 32_775, 32_776, 32_799, 32_800, 40_960, 40_961, m):
        for share in (0.0, 0.001, 0.4, 0.97):
            dd = d[:n].copy()
            dd[rng.random(n) < share, 1] = 0.0
            dd[[0, 7, 8, 31, 32, n // 4, n // 2, n - 1], 0] = 0.0
            ref = ora.intersect(o[:n], dd)
            out = dict(t=torch.full((n,), -7.0, dtype=torch.float64, device="cuda"),
                       uv=torch.full((n, 2), -7.0, dtype=torch.float64, device="cuda"),
                       normal=torch.full((n, 3), -7.0, dtype=torch.float64, device="cuda"),
                       prim=torch.full((n,), -7, dtype=torch.int32, device="cuda"),
                       geom=torch.full((n,), -7, dtype=torch.int32, device="cuda"),
                       hit=torch.full((n,), 7, dtype=torch.uint8, device="cuda"))
            got = to_numpy(scene.intersectN(torch.from_numpy(o[:n]).cuda(),
                                            torch.from_numpy(dd).cuda(), mode=mode, out=out))
            for k in ("prim", "geom"):
                got[k] = got[k].view(np.uint32)
            assert mismatches(got, ref) == [], (n, share)
    assert scene.check() == 0
    scene.close()
