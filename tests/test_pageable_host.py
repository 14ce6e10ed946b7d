"""Host-array batches from ordinary numpy arrays go through a ring of pinned blocks in chunks
(capi.cpp, run_staged).  At sizes on both sides of the chunk and of the ring, with every optional
array, with few, and with some arrays pinned, the results are those of device arrays."""
import threading

import numpy as np
import pytest

from blazert_b200 import workloads as W
from tests.helpers import mismatches, product_scene, to_numpy

pytestmark = pytest.mark.gpu

SIZES = [4097, (3 << 16) - 1, 3 << 16, (3 << 16) + 1, (1 << 18) - 5, 5 * (1 << 16) + 77, 400_003]


def _scene_and_rays():
    wl = W.mixed_primitives(n_rays=max(SIZES), n_spheres=500, n_cylinders=60, n_planes=30, seed=8)
    return product_scene(wl.scene), wl.rays


def _device(scene, o, d, lo, hi, any_hit=False):
    import torch

    dev = lambda a: None if a is None else torch.from_numpy(np.ascontiguousarray(a)).cuda()
    ref = to_numpy(scene.intersectN(dev(o), dev(d), dev(lo), dev(hi), any_hit=any_hit))
    for k in ("prim", "geom"):
        ref[k] = ref[k].view(np.uint32)
    return ref


@pytest.mark.parametrize("mode", ["fp64", "mixed"])
def test_pageable_batches_equal_device_batches(mode):
    import torch

    scene, R = _scene_and_rays()
    rng = np.random.default_rng(2)
    for n in SIZES:
        o, d = R.origins[:n], R.directions[:n]
        lo, hi = rng.choice([0.0, 5.0], n), rng.choice([np.inf, 80.0], n)
        assert mismatches(scene.intersectN(o, d, mode=mode), _device(scene, o, d, None, None)) == []
        ref = _device(scene, o, d, lo, hi, True)
        assert mismatches(scene.intersectN(o, d, lo, hi, mode=mode, any_hit=True), ref) == []
        few = scene.intersectN(o, d, lo, None, mode=mode, out=dict(hit=np.full(n, 9, np.uint8)))
        assert np.array_equal(few["hit"], _device(scene, o, d, lo, None)["hit"])
        # a caller that pinned its rays only
        po, pd = (torch.from_numpy(np.array(x)).pin_memory().numpy() for x in (o, d))
        assert mismatches(scene.intersectN(po, pd, lo, hi, mode=mode, any_hit=True), ref) == []
    assert scene.check() == 0
    scene.close()


def test_pageable_batches_from_threads():
    scene, R = _scene_and_rays()
    n = (3 << 16) + 1
    ref = _device(scene, R.origins[:n], R.directions[:n], None, None)
    bad = []

    def work():
        for _ in range(3):
            if mismatches(scene.intersectN(R.origins[:n], R.directions[:n]), ref):
                bad.append(1)
    th = [threading.Thread(target=work) for _ in range(4)]
    [t.start() for t in th]
    [t.join() for t in th]
    assert bad == []
    scene.close()
