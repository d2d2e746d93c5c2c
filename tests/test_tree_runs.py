"""The hierarchy's bottom-up construction around the runs of 512 positions that a
CTA joins by itself, from one leaf up, with distinct keys and with many equal ones
(coarse keys: whole runs of ties): nodes, parents and boxes of the oracle's
top-down construction and refit, bit for bit; and point location on it."""
import numpy as np
import pytest

import pmdas_gb300 as P
from oracle import pyoracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim,kind", [(3, P.SCENE_DISCS_MB), (4, P.SCENE_DISCS_DOF), (5, P.SCENE_DISCS_MBDOF),
                                      (6, P.SCENE_DISCS_MBDOF)])
def test_trees_of_growing_grids(cuda, dim, kind):
    torch = cuda
    W, H = 24, 16
    g = P.KDGrid(dim, 60000, 4, 0, 0, 0.0625, W, H)
    sc = P.Scene(kind, 4, 30, W, H, W, H)
    g.InitialSampling()
    sc.evaluate(g, 0, g.GetNumberOfSamples())
    sizes = []
    while g.GetNumberOfSamples() < 20000:
        st = g.dump_state()
        n = st["L"]
        sizes.append(n)
        for fine in (0, 1, 5):
            g.BuildHierarchy(fine)
            h = g.Hierarchy()
            sk, so = O.sort_pairs(O.leaf_keys(st["boxes"], dim, 0, 0, fine, W, H))
            ch, par = O.karras(sk)
            assert np.array_equal(h["keys"], sk) and np.array_equal(h["order"], so), (n, fine)
            assert np.array_equal(h["parents"], par), (n, fine)
            if n > 1:
                assert np.array_equal(h["children"], ch), (n, fine)
                assert np.array_equal(h["boxes"].view(np.uint32), O.refit(st["boxes"], so, ch).view(np.uint32)), (n, fine)
        pts = torch.rand(777, dim, device="cuda", generator=torch.Generator(device="cuda").manual_seed(n))
        pts[:, 0] *= W
        pts[:, 1] *= H
        assert np.array_equal(g.Locate(pts).cpu().numpy(), O.locate(st["boxes"], h["order"], pts.cpu().numpy())), n
        g.SamplingPass()
        a, b = g.GetNumberOfSamples(), g.GetNewSamples()
        sc.evaluate(g, a - b, b)
    assert sizes[0] == 1 and any(n > 1024 for n in sizes)
