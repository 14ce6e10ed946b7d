"""A batch through the pinned ring that times out keeps the ring while its work may still be queued.
The scene's next host-array call waits for that work, and gives the ring back with it."""
import os

import numpy as np
import pytest

import blazert_b200 as B
from blazert_b200 import workloads as W
from tests.helpers import mismatches, product_scene, to_numpy

pytestmark = pytest.mark.gpu


def test_a_timed_out_call_gives_the_ring_back_later():
    import torch

    lib = B.library()
    wl = W.mixed_primitives(n_rays=2_000_000, seed=33)
    R = wl.rays
    scene, other = product_scene(wl.scene), product_scene(wl.scene)
    o, d = torch.from_numpy(R.origins).cuda(), torch.from_numpy(R.directions).cuda()
    out = scene.intersectN(o, d)
    n = 400_000
    ref = {k: v[:n] for k, v in to_numpy(out).items()}
    for k in ("prim", "geom"):
        ref[k] = ref[k].view(np.uint32)
    assert mismatches(other.intersectN(R.origins[:n], R.directions[:n]), ref) == []
    assert lib.bzr_debug_ring_lent() == 0
    stream = torch.cuda.Stream()
    for _ in range(64):  # a hundred milliseconds of queued work before the call's own
        scene.intersectN(o, d, out=out, stream=stream)
    os.environ["BZR_TIMEOUT_MS"] = "1"
    try:
        with pytest.raises(B.BlazertError) as e:
            scene.intersectN(R.origins[:n], R.directions[:n])
        assert e.value.code == B.ETIMEOUT
    finally:
        del os.environ["BZR_TIMEOUT_MS"]
    assert lib.bzr_debug_ring_lent() == 1
    small = scene.intersectN(R.origins[:100], R.directions[:100])  # waits for the queued work
    assert mismatches(small, {k: v[:100] for k, v in ref.items()}) == []
    assert lib.bzr_debug_ring_lent() == 0
    for s in (other, scene):
        assert mismatches(s.intersectN(R.origins[:n], R.directions[:n]), ref) == []
    assert lib.bzr_debug_ring_lent() == 0
    scene.close()
    other.close()
