"""True errors of leaves that reach out of the scene's domain in one dimension each
(a loaded state whose boxes were moved: later shutter times, a wider lens, beside the
image; unbounded ones too), restated from the oracle's integrand, which tests every
disc, at the same points of the same random streams."""
import numpy as np
import pytest

import pmdas_gb300 as P
from oracle import pyoracle as O
from tests.test_shared_streams import _streams, _uniforms

pytestmark = pytest.mark.gpu
W, H = 20, 12


@pytest.mark.parametrize("kind,dim", [(P.SCENE_DISCS_MB, 3), (P.SCENE_DISCS_DOF, 4), (P.SCENE_DISCS_MBDOF, 5),
                                      (P.SCENE_DISCS_MBDOF, 6)])
def test_true_errors_of_leaves_outside_the_domain(cuda, kind, dim):
    torch = cuda
    samples, seed = 24, 5
    g = P.KDGrid(dim, 30000, 4, 0, 2, 0.25, W, H)
    sc = P.Scene(kind, 8, 200, W, H, W, H)
    g.InitialSampling()
    sc.evaluate(g, 0, g.GetNumberOfSamples())
    for _ in range(4):
        g.SamplingPass()
        n, new = g.GetNumberOfSamples(), g.GetNewSamples()
        sc.evaluate(g, n - new, new)
    st = g.dump_state()
    L = st["L"]
    b = st["boxes"].copy()
    for i in range(L):  # a quarter of the leaves stays, the others move along one dimension
        d = i % (dim + dim // 3 + 1)
        if d < dim:
            size = (W, H, 1, 1, 1, 1)[d]
            b[i, d], b[i, dim + d] = (np.float32(x + (4 * size if i % 2 else -4 * size)) for x in (b[i, d], b[i, dim + d]))
    g.load_state(dict(st, boxes=b))
    got = g.LeafTrueErrors(sc, samples=samples, seed=seed).cpu().numpy()
    u = _uniforms(_streams(seed, L), samples * dim).reshape(L, samples, dim)
    pts = (b[:, None, :dim] + u * (b[:, None, dim:] - b[:, None, :dim])).astype(np.float32)
    ref = O.evaluate_points(sc.export(), pts.reshape(-1, dim)).reshape(L, samples, 3).astype(np.float64).mean(1)
    valid = st["nodes"] >= 0
    v = st["values"][np.where(valid, st["nodes"], 0)]
    m = np.zeros((L, 3), np.float32)
    for k in range(4):
        m = np.where(valid[:, k, None], m + v[:, k], m)
    m = (m / valid.sum(1)[:, None].astype(np.float32)).astype(np.float64)
    # (the volume from the boxes as they are held: FP32 differences)
    vol = np.prod((b[:, dim:] - b[:, :dim]).astype(np.float64), axis=1)
    want = vol * (np.abs(m - ref) / np.sqrt(ref ** 2 + 1e-2)).sum(1)
    # FP32 means and volumes (D products), the result rounded to FP32
    assert np.allclose(got, want, rtol=1e-5, atol=1e-7 * float(vol.max()))


def test_true_errors_of_unbounded_leaves_return(cuda):
    g = P.KDGrid(5, 30000, 4, 0, 2, 0.25, W, H)
    sc = P.Scene(P.SCENE_DISCS_MBDOF, 8, 70, W, H, W, H)
    g.InitialSampling()
    sc.evaluate(g, 0, g.GetNumberOfSamples())
    st = g.dump_state()
    b = st["boxes"].copy()
    b[0, 5], b[1, 0], b[2, 2], b[3, 7] = np.inf, -np.inf, np.nan, np.nan
    whole = g.LeafTrueErrors(sc, samples=9, seed=2).cpu().numpy()
    g.load_state(dict(st, boxes=b))
    got = g.LeafTrueErrors(sc, samples=9, seed=2).cpu().numpy()
    assert not np.isfinite(got[:4]).any() and np.array_equal(got[4:], whole[4:])
