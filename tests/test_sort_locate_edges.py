"""Edges of the ordering kernels: the histogram of the radix sort where a thread's run of
keys and the grid's stride end, and point location at every dimension (a grid of one leaf
upwards) with points on faces, outside, infinite and not a number, against numpy and the
oracle."""
import numpy as np
import pytest

import pmdas_gb300 as P
from oracle import pyoracle as O


@pytest.mark.gpu
@pytest.mark.parametrize("n", [31, 255, 257, 2047, 2048, 2049, 608 * 2048 - 1, 608 * 2048 + 1])
@pytest.mark.parametrize("field", [(0, 64), (3, 30)])
def test_sort_at_histogram_edges(cuda, n, field):
    torch = cuda
    b, e = field
    rng = np.random.default_rng(n)
    k = rng.integers(0, 2 ** 64 - 1, size=n, dtype=np.uint64, endpoint=True)
    k[::3] = k[0]
    f = (k >> np.uint64(b)) & np.uint64((1 << (e - b)) - 1)
    want = np.argsort(f, kind="stable")
    ko, vo = P.radix_sort_pairs(torch.from_numpy(k.view(np.int64)).cuda(), None, b, e)
    assert np.array_equal(ko.cpu().numpy().view(np.uint64), k[want])
    assert np.array_equal(vo.cpu().numpy().view(np.uint32), want.astype(np.uint32))


@pytest.mark.gpu
@pytest.mark.parametrize("D,bpd,eib,passes", [(3, 0, 0, 0), (3, 0, 0, 1), (3, 1, 4, 5), (5, 1, 2, 3), (6, 1, 1, 3)])
def test_locate_at_every_dimension(cuda, D, bpd, eib, passes):
    torch = cuda
    W, H = 48, 32
    sx, sy = float(W), float(H)
    g = P.KDGrid(D, 60000, 4, bpd, eib, 0.25, sx, sy)
    scene = P.Scene(P.SCENE_DISCS_MB if D == 3 else P.SCENE_DISCS_MBDOF, 5, 32, sx, sy, W, H)
    g.InitialSampling()
    scene.evaluate(g, 0, g.GetNumberOfSamples())
    for _ in range(passes):
        g.SamplingPass()
        n, new = g.GetNumberOfSamples(), g.GetNewSamples()
        scene.evaluate(g, n - new, new)
    st = g.dump_state()
    g.BuildHierarchy(-1)
    order = g.Hierarchy()["order"]
    rng = np.random.default_rng(D)
    pts = rng.random((5000, D), dtype=np.float32)
    pts[:, 0] *= sx
    pts[:, 1] *= sy
    odd = np.tile(pts[:6], (3, 1))
    for i, v in enumerate((np.nan, np.inf, -np.inf)):
        for j in range(6):
            odd[6 * i + j, j % D] = v
    pts = np.concatenate([pts, st["boxes"][:2000, :D], st["boxes"][-2000:, D:], odd]).astype(np.float32)
    got = g.Locate(torch.from_numpy(pts).cuda()).cpu().numpy()
    assert np.array_equal(got, O.locate(st["boxes"], order, pts))
    assert (got[-18:] == -1).all() and (got[:5000] >= 0).all()
