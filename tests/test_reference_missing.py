"""Without the reference's sources a comparison with its own build is skipped, not failed, and the
GPU builder's trees are still compared: with the oracle's, which are the reference's node for node
(tests/test_oracle_pin.py, where its sources are present)."""
import unittest

import pytest

from blazert_b200 import BuildOptions
from blazert_b200 import workloads as W
from oracle.oracle import Oracle, RefScene
from tests.scenes import edge_case_scenes
from tests.test_gpu_builder import _cases, gpu_scene, same_tree_values


def test_a_missing_reference_build_skips(monkeypatch):
    spec = W.icosphere_pinhole(level=1, width=4, height=4).scene
    monkeypatch.setattr(RefScene, "_libs", {})
    with pytest.raises(unittest.SkipTest):
        RefScene(spec, flavour="of_no_build")
    with pytest.raises(RuntimeError):
        RefScene(spec, flavour="of_no_build")


OPTS = [dict(min_leaf=1, max_depth=28, bins=64), dict(min_leaf=8, max_depth=6, bins=16),
        dict(min_leaf=2, max_depth=40, bins=3), dict(min_leaf=4, max_depth=28, bins=256)]
SCENES = ([(name, wl.scene, {}) for name, wl in _cases()] +
          [(name, spec, {}) for name, spec, _ in edge_case_scenes()] +
          [(f"options{k}", W.mixed_primitives(n_rays=16, n_spheres=2000, n_cylinders=200,
                                              n_planes=40, seed=4).scene, o)
           for k, o in enumerate(OPTS)])


@pytest.mark.gpu
@pytest.mark.parametrize("name,spec,opts", SCENES, ids=[s[0] for s in SCENES])
def test_gpu_tree_is_the_oracle_tree(name, spec, opts):
    ora = Oracle(spec, **opts)
    g = gpu_scene(spec, BuildOptions(opts["min_leaf"], opts["max_depth"], opts["bins"])
                  if opts else None)
    for kind in spec.order:
        t = ora.tree(kind)
        if t is None or len(t["leaf"]) == 0:
            continue
        assert same_tree_values(g.tree(kind), t) is None, kind
