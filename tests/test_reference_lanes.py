"""The reference image at every number of lanes that may share a pixel: samples per pixel
around the lines of the rule, images below and above the sizes at which lanes are no
longer shared, scenes with culling lists, with few and with many primitives scanned in
full.  Some pixels are restated from the oracle's integrand at the same points of the
same random streams; the sums are of values below 16 in FP64, in any order, so 1e-12
bounds them."""
import numpy as np
import pytest

import pmdas_gb300 as P
from oracle import pyoracle as O
from tests.test_shared_streams import _streams, _uniforms

pytestmark = pytest.mark.gpu
SCENES = {"mb": (P.SCENE_DISCS_MB, 3, 40), "mbdof": (P.SCENE_DISCS_MBDOF, 5, 33), "light": (P.SCENE_DIRECT_LIGHT, 4, 31),
          "heavy": (P.SCENE_DIRECT_LIGHT, 4, 32)}


@pytest.mark.parametrize("size,stratas", [((13, 7), (2, 3, 4, 5, 6, 11, 12, 16, 17)), ((300, 200), (2, 3, 4, 6, 8, 16)),
                                          ((700, 500), (1, 2, 3, 16)), ((1100, 1000), (1, 2, 23))])
@pytest.mark.parametrize("kind", list(SCENES))
def test_reference_image_at_every_number_of_lanes(cuda, kind, size, stratas):
    scene, dim, prims = SCENES[kind]
    (W, H), seed, f = size, 99, np.float32
    sc = P.Scene(scene, 3, prims, W, H, W, H)
    rng = np.random.default_rng(W)
    px = np.unique(np.concatenate([[0, W - 1, W * H - 1], rng.integers(0, W * H, 40)]))
    for strata in stratas:
        if kind == "heavy" and strata > 16:
            continue
        got = sc.reference_image(W, H, spp=strata * strata, seed=seed).cpu().numpy().reshape(-1, 3)[px]
        u = _uniforms(_streams(seed, W * H)[px], strata * strata * dim).reshape(len(px), strata, strata, dim)
        i = np.arange(strata, dtype=f)
        pts = u.copy()
        pts[..., 0] = ((px % W).astype(f)[:, None, None] + (i[None, :, None] + u[..., 0]) / f(strata)) * (f(W) / f(W))
        pts[..., 1] = ((px // W).astype(f)[:, None, None] + (i[None, None, :] + u[..., 1]) / f(strata)) * (f(H) / f(H))
        vals = O.evaluate_points(sc.export(), pts.reshape(-1, dim)).reshape(len(px), strata * strata, 3)
        want = vals.astype(np.float64).sum(1) * (1.0 / (float(strata) * float(strata)))
        assert np.allclose(got, want, rtol=1e-12, atol=1e-12), strata
