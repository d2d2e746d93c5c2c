"""The device-side render loops over scenes without culling lists, around the number of
primitives from which the values kernel takes more CTAs and up to the largest scene, and a
batch that mixes them with culled scenes of the same dimension (each kind has an instance
of the values kernel of its own): bit for bit the host loop's state."""
import pytest

import pmdas_gb300 as P
from tests.parity import assert_states_equal, rel_close

pytestmark = pytest.mark.gpu
W, H, SPP = 53, 31, 14
KEYS = ("coords", "values", "nodes", "boxes", "errors", "seeds")
LIGHT, DOF, MB = P.SCENE_DIRECT_LIGHT, P.SCENE_DISCS_DOF, P.SCENE_DISCS_MB


def _make(dim, kind, prims, arith, k=0):
    g = P.KDGrid(dim, 3 * SPP * W * H, 4, 0, 3, 0.25, W, H, arith=arith)
    return g, P.Scene(kind, 9 + k, prims, W, H, W, H)


def _host(torch, dim, kind, prims, arith, k=0):
    g, s = _make(dim, kind, prims, arith, k)
    px = torch.zeros(H, W, 4, device="cuda")
    st = P.render(g, s, SPP * W * H, px, W, H)
    return g.dump_state(), px.cpu().numpy(), st


def _same(g, px, st, want, what):
    assert (st.numberOfSamples, st.numberOfNodes, st.passes) == (want[2].numberOfSamples, want[2].numberOfNodes,
                                                                want[2].passes)
    assert_states_equal(g.dump_state(), want[0], keys=KEYS, what=what)
    ok, worst = rel_close(px.cpu().numpy(), want[1])
    assert ok, worst


@pytest.mark.parametrize("arith", [P.ARITH_REFERENCE, P.ARITH_IEEE])
@pytest.mark.parametrize("dim", [4, 5, 6])
@pytest.mark.parametrize("prims", [1, 31, 127, 128, 1023, 1024])
def test_full_scan_renders_equal_the_host_loop(cuda, prims, dim, arith):
    torch = cuda
    g, s = _make(dim, LIGHT, prims, arith)
    px = torch.zeros(H, W, 4, device="cuda")
    st = P.render_graph(g, s, SPP * W * H, px, W, H)
    _same(g, px, st, _host(torch, dim, LIGHT, prims, arith), "graph")


@pytest.mark.parametrize("learned", [False, True])
@pytest.mark.parametrize("scenes", [((4, DOF, 70), (4, LIGHT, 200), (4, DOF, 0), (4, MB, 40), (4, LIGHT, 4)),
                                    ((3, MB, 9), (4, LIGHT, 1024), (5, MB, 0), (5, DOF, 33), (6, LIGHT, 2)),
                                    ((4, LIGHT, 3), (4, LIGHT, 300))])
def test_batches_of_both_kinds_equal_the_host_loop(cuda, scenes, learned):
    torch = cuda
    made = [_make(*c, P.ARITH_REFERENCE, k) for k, c in enumerate(scenes)]
    if learned:
        for g, _ in made:
            g.LearnedEnable(seed=3)
    px = [torch.zeros(H, W, 4, device="cuda") for _ in scenes]
    n = len(scenes)
    batch = P.Batch([g for g, _ in made], [s for _, s in made], [SPP * W * H] * n, px, [W] * n, [H] * n)
    for render in (batch.render, batch.render_stepped):
        stats = render()
        for k, c in enumerate(scenes):
            if learned:  # the learned loop of one image
                g, s = _make(*c, P.ARITH_REFERENCE, k)
                g.LearnedEnable(seed=3)
                one = torch.zeros(H, W, 4, device="cuda")
                st = P.render_graph(g, s, SPP * W * H, one, W, H)
                want = (g.dump_state(), one.cpu().numpy(), st)
            else:
                want = _host(torch, *c, P.ARITH_REFERENCE, k)
            _same(made[k][0], px[k], stats[k], want, f"image {k}")
