"""Small batches (trace_small.cu) take one launch for every kind.  At sizes on both sides of its
grid's steps (a ray alone in its warp, the last block ragged, the largest batch it takes) the
results are the oracle's, from device and from host arrays, with every optional array and with
one."""
import numpy as np
import pytest

from blazert_b200 import workloads as W
from oracle.oracle import Oracle
from tests.helpers import mismatches, product_scene, to_numpy

pytestmark = pytest.mark.gpu


def _spec(kinds):
    spec = W.mixed_primitives(n_rays=1, n_spheres=400, n_cylinders=150, n_planes=80, seed=3).scene
    v, f = W.icosphere(3)
    out = W.SceneSpec()
    for k in kinds:
        out.add_mesh(40.0 * v, f) if k == "mesh" else getattr(out, "add_" + k)(
            *getattr(spec, k).values())
    return out


def _rays(n, seed):
    rng = np.random.default_rng(seed)
    o, d = rng.uniform(-120.0, 120.0, (n, 3)), rng.standard_normal((n, 3))
    d[::5] = rng.permuted(np.tile([0.0, 0.0, -1.0], (len(d[::5]), 1)), axis=1)  # axis-parallel
    return o, d, rng.choice([0.0, -3.0, 10.0], n), rng.choice([np.inf, 60.0, 0.0], n)


@pytest.mark.parametrize("any_hit", [False, True], ids=["closest", "any"])
@pytest.mark.parametrize("kinds", [["mesh"], ["cylinders", "spheres"],
                                   ["planes", "spheres", "cylinders"],
                                   ["spheres", "planes", "mesh", "cylinders"]],
                         ids=lambda k: "-".join(k))
def test_small_batches_equal_oracle(kinds, any_hit):
    import torch

    spec = _spec(kinds)
    scene, ora = product_scene(spec), Oracle(spec)
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    for n in (1, 2, 31, 33, 739, 741, 1481, 4096, 4097, 16383, 16384, 16385):
        o, d, tmin, tmax = _rays(n, n)
        for lo, hi in ((None, None), (tmin, tmax)):
            ref = ora.intersect(o, d, lo, hi, any_hit=any_hit)
            a = [None if x is None else dev(x) for x in (o, d, lo, hi)]
            assert mismatches(scene.intersectN(*a, any_hit=any_hit), ref) == [], (n, "device")
            got = scene.intersectN(o, d, lo, hi, any_hit=any_hit)
            assert mismatches(got, ref) == [], (n, "host")
        only = scene.intersectN(dev(o), dev(d), out=dict(prim=torch.empty(n, dtype=torch.int32,
                                                                         device="cuda")))
        ref = ora.intersect(o, d)
        assert np.array_equal(only["prim"].cpu().numpy().view(np.uint32), ref["prim"])
        only = scene.intersectN(o, d, out=dict(hit=np.full(n, 7, np.uint8)))
        assert np.array_equal(only["hit"], ref["hit"])
    assert scene.check() == 0
    scene.close()


def test_small_batches_on_many_streams():
    """Calls on several streams and host calls from several threads at once share no state."""
    import threading

    import torch

    spec = _spec(["spheres", "planes", "mesh", "cylinders"])
    scene, ora = product_scene(spec), Oracle(spec)
    jobs = [_rays(n, 100 + n)[:2] for n in (5, 700, 3000, 9000)]
    refs = [ora.intersect(o, d) for o, d in jobs]
    streams = [torch.cuda.Stream() for _ in jobs]
    devs = [[torch.from_numpy(x).cuda() for x in j] for j in jobs]
    torch.cuda.synchronize()
    for _ in range(5):
        outs = [scene.intersectN(o, d, stream=s) for (o, d), s in zip(devs, streams)]
        torch.cuda.synchronize()
        for out, ref in zip(outs, refs):
            assert mismatches(to_numpy(out), {k: v for k, v in ref.items()}) == []
    bad = []

    def work(j):
        for _ in range(10):
            o, d = jobs[j]
            if mismatches(scene.intersectN(o[:3000], d[:3000]),
                          {k: v[:3000] for k, v in refs[j].items() if hasattr(v, "shape")}):
                bad.append(j)
    th = [threading.Thread(target=work, args=(j,)) for j in range(len(jobs))]
    [t.start() for t in th]
    [t.join() for t in th]
    assert bad == []
    assert scene.check() == 0
    scene.close()


def test_a_new_scene_does_not_see_an_earlier_scenes_flag():
    """The flag that ends a small host-array call lies in pinned memory that a closed scene may
    have used for its own: the first calls of a new scene wait for their own results."""
    import blazert_b200 as B

    rng = np.random.default_rng(4)
    for k in range(12):
        c, r = rng.uniform(-1.0, 1.0, (50, 3)), rng.uniform(0.1, 0.4, 50)
        spec = W.SceneSpec().add_spheres(c, r)
        scene, ora = product_scene(spec), Oracle(spec)
        for _ in range(3):
            o = 4.0 * W._unit_sphere(rng, 1)
            d = rng.uniform(-0.5, 0.5, (1, 3)) - o
            ref = ora.intersect(o, d)
            hit, rh = scene.intersect1(B.Ray(o[0], d[0]))
            assert hit == bool(ref["hit"][0]) and rh.prim_id == ref["prim"][0], k
            assert not hit or rh.hit_distance == ref["t"][0]
        scene.close()
