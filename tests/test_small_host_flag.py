"""Small host-array calls end on a flag that the kernel raises in pinned memory: whatever the number
of blocks (one, a few, a full wave), the results and the error word that the host then reads are
the call's own, call after call with changing inputs."""
import numpy as np
import pytest

from blazert_b200 import workloads as W
from oracle.oracle import Oracle
from tests.helpers import mismatches, product_scene

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kinds", [["spheres"], ["spheres", "planes", "cylinders"]],
                         ids=lambda k: "-".join(k))
def test_results_are_there_when_the_flag_is(kinds):
    full = W.mixed_primitives(n_rays=1, n_spheres=300, n_cylinders=60, n_planes=30, seed=5).scene
    spec = W.SceneSpec()
    for k in kinds:
        getattr(spec, "add_" + k)(*getattr(full, k).values())
    scene, ora = product_scene(spec), Oracle(spec)
    rng = np.random.default_rng(8)
    pool = [(rng.uniform(-120.0, 120.0, (4096, 3)), rng.standard_normal((4096, 3)))
            for _ in range(4)]
    refs = [ora.intersect(o, d) for o, d in pool]
    for n in (1, 2, 33, 700, 4096):
        for rep in range(200 if n < 700 else 60):
            (o, d), ref = pool[rep % 4], refs[rep % 4]
            out = scene.intersectN(o[:n], d[:n])  # raises if an error word is set
            assert mismatches(out, {k: v[:n] for k, v in ref.items() if hasattr(v, "shape")}) == []
    scene.close()
