"""The integrand over the culled disc lists at list lengths around their packing
(two discs per word, 32 per step of the build) and at the largest scene: the
oracle's full scan bit for bit, image corners and edges included."""
import numpy as np
import pytest

import pmdas_gb300 as P
from oracle import pyoracle as O
from tests.test_integrand import gpu_evaluate, points

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("count", [0, 1, 2, 3, 31, 32, 33, 64, 1024])
@pytest.mark.parametrize("kind,dim", [(P.SCENE_DISCS_MB, 3), (P.SCENE_DISCS_DOF, 4), (P.SCENE_DISCS_MBDOF, 5)])
def test_lists_of_every_length(cuda, kind, dim, count):
    W, H = 48, 33
    sc = P.Scene(kind, 7, count, W, H, W, H)
    pts = points(dim, 1 << 15, W, H, count)
    got = gpu_evaluate(sc, pts)
    want = O.evaluate_points(sc.export(), pts)
    assert np.array_equal(got.view(np.uint32), want.view(np.uint32))
    sc.close()
