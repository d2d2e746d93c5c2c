"""True errors of leaves at every number of lanes that may share a leaf: numbers of leaves
and of points around the lines of the rule, scenes with culling lists, with few and with
many primitives scanned in full, restated from the oracle's integrand at the same points
of the same random streams."""
import numpy as np
import pytest

import pmdas_gb300 as P
from oracle import pyoracle as O
from tests.test_shared_streams import _streams, _uniforms

pytestmark = pytest.mark.gpu
SCENES = [(3, P.SCENE_DISCS_MB, 40), (4, P.SCENE_DIRECT_LIGHT, 31), (4, P.SCENE_DIRECT_LIGHT, 32),
          (5, P.SCENE_DISCS_MBDOF, 33), (6, P.SCENE_DIRECT_LIGHT, 40)]


@pytest.mark.parametrize("dim,kind,prims", SCENES)
def test_true_errors_at_every_number_of_lanes(cuda, dim, kind, prims):
    torch = cuda
    W, H, seed = 20, 12, 5
    g = P.KDGrid(dim, 30000, 4, 0, 2, 0.25, W, H)
    sc = P.Scene(kind, 8, prims, W, H, W, H)
    g.InitialSampling()
    sc.evaluate(g, 0, g.GetNumberOfSamples())
    for _ in range(3):
        g.SamplingPass()
        n, new = g.GetNumberOfSamples(), g.GetNewSamples()
        sc.evaluate(g, n - new, new)
    st = g.dump_state()
    L, b = st["L"], st["boxes"]
    u = _uniforms(_streams(seed, L), 33 * dim).reshape(L, 33, dim)
    pts = (b[:, None, :dim] + u * (b[:, None, dim:] - b[:, None, :dim])).astype(np.float32)
    vals = O.evaluate_points(sc.export(), pts.reshape(-1, dim)).reshape(L, 33, 3).astype(np.float64)
    valid = st["nodes"] >= 0
    v = st["values"][np.where(valid, st["nodes"], 0)]
    m = np.zeros((L, 3), np.float32)
    for k in range(4):
        m = np.where(valid[:, k, None], m + v[:, k], m)
    m = (m / valid.sum(1)[:, None].astype(np.float32)).astype(np.float64)
    vol = np.prod((b[:, dim:] - b[:, :dim]).astype(np.float64), axis=1)
    rng = np.random.default_rng(dim)
    for count in (1, 31, 8192, 8193, 65536, 65537, 131072, 131073):
        pick = rng.integers(0, L, count).astype(np.int32)
        for samples in (1, 3, 4, 7, 8, 15, 16, 31, 32, 33):
            ref = vals[:, :samples].mean(1)
            want = (vol * (np.abs(m - ref) / np.sqrt(ref ** 2 + 1e-2)).sum(1))[pick]
            got = g.LeafTrueErrors(sc, samples=samples, seed=seed, leaves=torch.from_numpy(pick).cuda()).cpu().numpy()
            # FP32 means and volumes (D products), the result rounded to FP32
            assert np.allclose(got, want, rtol=1e-5, atol=1e-7 * float(vol.max())), (count, samples)
