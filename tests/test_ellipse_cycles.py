"""The cylinder distance's ellipse search skips whole periods once a value of the search comes
back (distance_core.cuh, ellipse_search_step).  Its results stay the oracle's, which steps
through all 100, bit for bit: for searches that converge, that end on a fixed point, and that
end in a cycle of several values."""
import numpy as np
import pytest

from blazert_b200 import workloads as W
from oracle.oracle import Oracle
from tests.emu.emu import EmuScene
from tests.helpers import bits_equal


@pytest.mark.parametrize("ratio", [1.0, 1.0 + 1e-12, 1.7, 30.0, 1e-3])
@pytest.mark.parametrize("scale", [1e-6, 1.0, 1e7])
def test_search_results_are_the_full_searchs(ratio, scale):
    rng = np.random.default_rng(17)
    n, m = 40, 6000
    a = scale * rng.uniform(0.1, 1.0, n)
    spec = W.SceneSpec().add_cylinders(scale * rng.uniform(-1.0, 1.0, (n, 3)), a, ratio * a,
                                       scale * rng.uniform(0.5, 5.0, n),
                                       W.rotation_to(W._unit_sphere(rng, n)))
    ids = rng.integers(0, n, m).astype(np.uint32)
    # near the surface (few steps), around it and far away (the derivative's rounding never
    # falls below the stopping rule: fixed points and cycles)
    reach = scale * 10.0 ** rng.uniform(-3.0, 5.0, (m, 1))
    pts = spec.cylinders["centers"][ids] + reach * rng.standard_normal((m, 3))
    want, _ = Oracle(spec).distance_to_surface("cylinders", ids, pts)
    got, _ = EmuScene(spec).distance_to_surface("cylinders", ids, pts)
    assert bits_equal(got, want)
