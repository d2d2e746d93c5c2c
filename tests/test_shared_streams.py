"""The reference image and the true errors, whose samples several lanes share:
every scene kind, samples per pixel below and above a lane's share, image and
leaf counts that leave lanes without a pixel or leaf.  Both are restated from
the oracle's integrand at the same points of the same random streams; the image
sums values below 16 in FP64, in any order, so 1e-12 bounds it."""
import numpy as np
import pytest

import pmdas_gb300 as P
from oracle import pyoracle as O

pytestmark = pytest.mark.gpu

KINDS = {"mb": (P.SCENE_DISCS_MB, 3, 40), "dof": (P.SCENE_DISCS_DOF, 4, 70), "mbdof": (P.SCENE_DISCS_MBDOF, 5, 33),
         "light": (P.SCENE_DIRECT_LIGHT, 4, 4), "empty": (P.SCENE_DISCS_DOF, 4, 0)}
A, C = np.uint64(6364136223846793005), np.uint64(1442695040888963407)


def _uniforms(states, n):
    """n successive 24-bit uniforms of every stream: [streams, n] float32."""
    out = np.empty((len(states), n), np.float32)
    s = states.copy()
    with np.errstate(over="ignore"):
        for k in range(n):
            s = s * A + C
            out[:, k] = (s >> np.uint64(40)).astype(np.float32) * np.float32(1 / 16777216)
    return out


def _streams(seed, n):
    with np.errstate(over="ignore"):
        return np.uint64(seed) ^ (np.uint64(0x9E3779B97F4A7C15) * (np.arange(n, dtype=np.uint64) + np.uint64(1)))


@pytest.mark.parametrize("strata", [1, 2, 3, 7, 8, 9])
@pytest.mark.parametrize("kind", list(KINDS))
def test_reference_image_sums_the_stream_of_each_pixel(cuda, kind, strata):
    scene, dim, prims = KINDS[kind]
    W, H, seed = 13, 7, 99
    sc = P.Scene(scene, 3, prims, W, H, W, H)
    got = sc.reference_image(W, H, spp=strata * strata, seed=seed).cpu().numpy()
    u = _uniforms(_streams(seed, W * H), strata * strata * dim).reshape(W * H, strata, strata, dim)
    f = np.float32
    i = np.arange(strata, dtype=f)
    p = np.arange(W * H)
    pts = u.copy()
    pts[..., 0] = ((p % W).astype(f)[:, None, None] + (i[None, :, None] + u[..., 0]) / f(strata)) * (f(W) / f(W))
    pts[..., 1] = ((p // W).astype(f)[:, None, None] + (i[None, None, :] + u[..., 1]) / f(strata)) * (f(H) / f(H))
    vals = O.evaluate_points(sc.export(), pts.reshape(-1, dim)).reshape(W * H, strata * strata, 3).astype(np.float64)
    want = (vals.sum(1) * (1.0 / (float(strata) * float(strata)))).reshape(H, W, 3)
    assert np.allclose(got, want, rtol=1e-12, atol=1e-12)


@pytest.mark.parametrize("samples", [1, 7, 8, 20])
@pytest.mark.parametrize("dim", [3, 4, 5, 6])
def test_true_errors_of_listed_leaves_equal_those_of_all(cuda, dim, samples):
    torch = cuda
    scene = {3: "mb", 4: "light", 5: "mbdof", 6: "mbdof"}[dim]
    kind, _, prims = KINDS[scene]
    W, H = 20, 12
    g = P.KDGrid(dim, 30000, 4, 0, 2, 0.25, W, H)
    sc = P.Scene(kind, 8, prims, W, H, W, H)
    g.InitialSampling()
    sc.evaluate(g, 0, g.GetNumberOfSamples())
    for _ in range(3):
        g.SamplingPass()
        n, new = g.GetNumberOfSamples(), g.GetNewSamples()
        sc.evaluate(g, n - new, new)
    st = g.dump_state()
    L = st["L"]
    whole = g.LeafTrueErrors(sc, samples=samples, seed=5).cpu().numpy()
    b = st["boxes"]
    u = _uniforms(_streams(5, L), samples * dim).reshape(L, samples, dim)
    pts = (b[:, None, :dim] + u * (b[:, None, dim:] - b[:, None, :dim])).astype(np.float32)
    ref = O.evaluate_points(sc.export(), pts.reshape(-1, dim)).reshape(L, samples, 3).astype(np.float64).mean(1)
    valid = st["nodes"] >= 0
    v = st["values"][np.where(valid, st["nodes"], 0)]
    m = np.zeros((L, 3), np.float32)
    for k in range(4):
        m = np.where(valid[:, k, None], m + v[:, k], m)
    m = (m / valid.sum(1)[:, None].astype(np.float32)).astype(np.float64)
    vol = np.prod((b[:, dim:] - b[:, :dim]).astype(np.float64), axis=1)
    want = vol * (np.abs(m - ref) / np.sqrt(ref ** 2 + 1e-2)).sum(1)
    # FP32 means and volumes (D products), the result rounded to FP32
    assert np.allclose(whole, want, rtol=1e-5, atol=1e-7 * float(vol.max()))
    pick = torch.tensor([L - 1, 0, L // 2, 0, 3], dtype=torch.int32, device="cuda")
    some = g.LeafTrueErrors(sc, samples=samples, seed=5, leaves=pick).cpu().numpy()
    assert np.array_equal(some, whole[pick.cpu().numpy()])
