"""Calls that run at the same time use device words of their own: a captured call replayed beside
direct ones on other streams, and more direct calls in flight than there are slots.  Every call
has rays that its wide pass hands on through the lists in those words."""
import numpy as np
import pytest

from oracle.oracle import Oracle
from tests.helpers import mismatches, product_scene, uncovered_workload

pytestmark = pytest.mark.gpu


def _outputs(n, dev):
    import torch

    f64 = torch.float64
    return dict(t=torch.zeros(n, dtype=f64, device=dev),
                uv=torch.zeros((n, 2), dtype=f64, device=dev),
                normal=torch.zeros((n, 3), dtype=f64, device=dev),
                prim=torch.zeros(n, dtype=torch.int32, device=dev),
                geom=torch.zeros(n, dtype=torch.int32, device=dev),
                hit=torch.zeros(n, dtype=torch.uint8, device=dev))


def _same(out, ref):
    out = {k: v.cpu().numpy() for k, v in out.items() if not k.startswith("_")}
    for k in ("prim", "geom"):
        out[k] = out[k].view(np.uint32)
    return mismatches(out, ref) == []


@pytest.mark.parametrize("mode", ["fp64", "mixed"])
def test_captured_and_direct_calls_share_no_words(mode):
    import torch

    dev = torch.device("cuda", 0)
    wl, _ = uncovered_workload(60_000, 31)
    R = wl.rays
    scene, ora = product_scene(wl.scene), Oracle(wl.scene)
    sizes = (60_000, 25_000, 31_003)  # all above what the one launch of small batches takes
    refs = [ora.intersect(R.origins[:n], R.directions[:n]) for n in sizes]
    args = [[torch.from_numpy(np.ascontiguousarray(a[:n])).to(dev)
             for a in (R.origins, R.directions)] for n in sizes]
    captured = _outputs(sizes[0], dev)
    scene.intersectN(*args[0], mode=mode, out=captured)  # warm
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        scene.intersectN(*args[0], mode=mode, out=captured)
    streams = [torch.cuda.Stream() for _ in range(4)]
    outs = [_outputs(sizes[1 + k % 2], dev) for k in range(4)]
    for rep in range(3):
        for v in [captured[k] for k in captured if not k.startswith("_")]:
            v.fill_(7)
        torch.cuda.synchronize()
        for j in range(75):  # 300 direct calls beside the replays: more than the slots
            if j % 5 == 0:
                graph.replay()
            for k, st in enumerate(streams):
                scene.intersectN(*args[1 + k % 2], mode=mode, out=outs[k], stream=st)
        torch.cuda.synchronize()
        assert _same(captured, refs[0]), rep
        for k in range(4):
            assert _same(outs[k], refs[1 + k % 2]), (rep, k)
    assert scene.check() == 0
    scene.close()
