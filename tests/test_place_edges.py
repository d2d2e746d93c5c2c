"""The adaptive pass at the edges of its 32-leaf groups: grids that start from
one leaf and grow through partial groups, groups in which every leaf splits
(alpha 0 accepts every leaf) and mixed ones, in every dimension, bit for bit
against the CPU oracle."""
import pytest

import pmdas_gb300 as P
from oracle import pyoracle as O
from tests.parity import assert_states_equal

pytestmark = pytest.mark.gpu

SCENE_OF = {3: P.SCENE_DISCS_MB, 4: P.SCENE_DISCS_DOF, 5: P.SCENE_DISCS_MBDOF, 6: P.SCENE_DISCS_MBDOF}


@pytest.mark.parametrize("alpha", [0.0, 0.25])
@pytest.mark.parametrize("cells", [(0, 0), (0, 1), (1, 0)])
@pytest.mark.parametrize("dim", [3, 4, 5, 6])
def test_passes_through_partial_and_whole_groups(cuda, dim, cells, alpha):
    bpd, eib = cells
    W, H, most, passes = 24, 16, 40000, 9
    g = P.KDGrid(dim, most, 4, bpd, eib, alpha, W, H, arith=P.ARITH_IEEE)
    sc = P.Scene(SCENE_OF[dim], 5, 24, W, H, W, H)
    o = O.OracleGrid(dim, most, 4, bpd, eib, alpha, W, H)
    desc = sc.export()
    g.InitialSampling()
    o.initial_sampling()
    sc.evaluate(g, 0, g.GetNumberOfSamples())
    o.evaluate(desc, 0, o.N)
    for k in range(passes):
        g.SamplingPass()
        o.sampling_pass()
        n, new = g.GetNumberOfSamples(), g.GetNewSamples()
        sc.evaluate(g, n - new, new)
        o.evaluate(desc, o.N - o.newN, o.newN)
        assert_states_equal(g.dump_state(), o.dump_state(),
                            keys=("coords", "values", "nodes", "boxes", "errors", "seeds"), what=f"pass {k}")
    assert g.Validate()
