"""A device-side render after its scene was destroyed and another one created, which
the allocator mostly places at the address of the first: the render is of the new
scene, bit for bit the host loop's on a fresh grid."""
import numpy as np
import pytest

import pmdas_gb300 as P
from tests.parity import assert_states_equal, rel_close

pytestmark = pytest.mark.gpu
W, H, BUDGET = 40, 24, 6000
DOF, MB, LIGHT = P.SCENE_DISCS_DOF, P.SCENE_DISCS_MB, P.SCENE_DIRECT_LIGHT


def _grid():
    return P.KDGrid(4, 20000, 4, 0, 3, 0.25, W, H)


@pytest.mark.parametrize("host", [False, True])
@pytest.mark.parametrize("first,second", [((DOF, 500), (DOF, 9)), ((DOF, 9), (MB, 300)), ((LIGHT, 4), (DOF, 70)),
                                          ((MB, 40), (LIGHT, 3)), ((DOF, 64), (DOF, 0))])
def test_render_of_a_scene_at_a_destroyed_ones_address(cuda, first, second, host):
    torch = cuda
    g = _grid()
    px = torch.zeros(H, W, 4, device="cuda")
    hpx = np.zeros((H, W, 4), np.float32)

    def render(s):
        if host:
            P.render_host(g, s, BUDGET, hpx, W, H)
            return hpx.copy()
        P.render_graph(g, s, BUDGET, px, W, H)
        return px.cpu().numpy()

    def check(s):
        img = render(s)
        other, ref = _grid(), torch.zeros(H, W, 4, device="cuda")
        P.render(other, s, BUDGET, ref, W, H)
        assert_states_equal(g.dump_state(), other.dump_state(),
                            keys=("coords", "values", "nodes", "boxes", "errors", "seeds"))
        ok, worst = rel_close(img, ref.cpu().numpy())
        assert ok, worst

    a = P.Scene(first[0], 1, first[1], W, H, W, H)
    check(a)
    address = a.handle.value
    a.close()
    scenes = []
    for _ in range(64):  # until one lies at the address (the others stay alive meanwhile)
        scenes.append(P.Scene(second[0], 2, second[1], W, H, W, H))
        if scenes[-1].handle.value == address:
            break
    check(scenes[-1])
