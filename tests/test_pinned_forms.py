"""Large batches from host arrays of which some are pinned: the pinned ones are copied straight, the
others through the ring, with every combination of optional arrays the same results."""
import numpy as np
import pytest

from blazert_b200 import workloads as W
from tests.helpers import mismatches, product_scene, to_numpy

pytestmark = pytest.mark.gpu

NAMES = ("o", "d", "tmin", "tmax", "t", "uv", "normal", "prim", "geom", "hit")
FORMS = [("o", "d"), ("t", "uv", "normal", "prim", "geom", "hit"), ("o",), ("hit",), ("tmin",),
         ("o", "tmax", "uv", "hit"), ("d", "tmin", "t", "prim"), NAMES[:4], NAMES[:9], NAMES, ()]


@pytest.mark.parametrize("pinned", FORMS, ids=lambda f: "-".join(f) or "none")
@pytest.mark.parametrize("n", [3 << 16, (5 << 16) + 77])
def test_some_arrays_pinned(n, pinned):
    import torch

    wl = W.mixed_primitives(n_rays=n, n_spheres=200, n_cylinders=30, n_planes=20, seed=6)
    scene = product_scene(wl.scene)
    rng = np.random.default_rng(n)
    pin = lambda a: torch.from_numpy(np.ascontiguousarray(a)).pin_memory().numpy()
    a = dict(o=wl.rays.origins, d=wl.rays.directions, tmin=rng.choice([0.0, 5.0], n),
             tmax=rng.choice([np.inf, 90.0], n), t=np.zeros(n), uv=np.zeros((n, 2)),
             normal=np.zeros((n, 3)), prim=np.zeros(n, np.uint32), geom=np.zeros(n, np.uint32),
             hit=np.zeros(n, np.uint8))
    a = {k: pin(v) if k in pinned else np.array(v) for k, v in a.items()}
    ref = to_numpy(scene.intersectN(*(torch.from_numpy(a[k]).cuda() for k in NAMES[:4])))
    for k in ("prim", "geom"):
        ref[k] = ref[k].view(np.uint32)
    out = {k: a[k] for k in NAMES[4:]}
    assert mismatches(scene.intersectN(*(a[k] for k in NAMES[:4]), out=out), ref) == []
    # without distances (the passes carry them on the device) and with one array only
    for keep in (("prim", "hit"), ("normal",)):
        for k in NAMES[4:]:
            a[k][...] = 9
        got = scene.intersectN(*(a[k] for k in NAMES[:4]), out={k: a[k] for k in keep})
        for k in keep:
            x, y = np.ascontiguousarray(got[k]), ref[k]
            assert np.array_equal(x.view(np.uint8).reshape(-1), np.ascontiguousarray(y).view(
                np.uint8).reshape(-1)), k
    assert scene.check() == 0
    scene.close()
