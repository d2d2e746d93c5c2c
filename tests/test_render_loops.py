"""The device-side render loops (which evaluate samples and compute the errors of
split children where they place them) against the host loop: state bit for bit,
image within the order of its float additions, in every dimension and scene kind,
from one initial leaf up, with every leaf accepted (alpha 0), with no pass at all,
and a pass of the drop-in calls after the render."""
import numpy as np
import pytest

import pmdas_gb300 as P
from tests.parity import assert_states_equal, rel_close

pytestmark = pytest.mark.gpu
KEYS = ("coords", "values", "nodes", "boxes", "errors", "seeds")
KINDS = {"mb": (P.SCENE_DISCS_MB, 40), "dof": (P.SCENE_DISCS_DOF, 70), "mbdof": (P.SCENE_DISCS_MBDOF, 33),
         "light": (P.SCENE_DIRECT_LIGHT, 4), "empty": (P.SCENE_DISCS_DOF, 0)}
CASES = [(3, "mb"), (4, "mb"), (4, "dof"), (4, "light"), (4, "empty"), (5, "mbdof"), (5, "light"), (6, "mbdof"), (6, "dof")]


def _make(dim, kind, cells, alpha, arith, W, H, most):
    scene, prims = KINDS[kind]
    g = P.KDGrid(dim, most, 4, cells[0], cells[1], alpha, W, H, arith=arith)
    return g, P.Scene(scene, 9, prims, W, H, W, H)


@pytest.mark.parametrize("arith", [P.ARITH_REFERENCE, P.ARITH_IEEE])
@pytest.mark.parametrize("cells,alpha,spp", [((0, 0), 0.0, 40), ((0, 2), 0.25, 9), ((1, 1), 0.0625, 20), ((1, 2), 0.25, 0.1)])
@pytest.mark.parametrize("dim,kind", CASES)
def test_render_loops_equal_the_host_loop(cuda, dim, kind, cells, alpha, spp, arith):
    torch = cuda
    W, H = 37, 21
    budget = int(spp * W * H)
    most = 3 * max(budget, 4 * ((1 << (cells[0] * dim)) << (2 * cells[1]))) + 64
    px = [torch.zeros(H, W, 4, device="cuda") for _ in range(3)]
    a, sa = _make(dim, kind, cells, alpha, arith, W, H, most)
    st = P.render(a, sa, budget, px[0], W, H)
    want = a.dump_state()
    b, sb = _make(dim, kind, cells, alpha, arith, W, H, most)
    c, sc = _make(dim, kind, cells, alpha, arith, W, H, most)
    batch = P.Batch([c], [sc], [budget], [px[2]], [W], [H])
    renders = (lambda: P.render_graph(b, sb, budget, px[1], W, H), lambda: batch.render()[0])
    for k, (g, render) in enumerate(zip((b, c), renders)):
        for again in range(2):
            got = render()
            assert (got.numberOfSamples, got.numberOfNodes, got.passes) == (st.numberOfSamples, st.numberOfNodes, st.passes)
            assert_states_equal(g.dump_state(), want, keys=KEYS, what=f"loop {k}, render {again}")
            ok, worst = rel_close(px[1 + k].cpu().numpy(), px[0].cpu().numpy())
            assert ok, worst
        assert g.GetGError() == a.GetGError() and g.pass_stats() == a.pass_stats()
    # a pass of the drop-in calls on the finished renders
    for g, s in ((a, sa), (b, sb), (c, sc)):
        g.SamplingPass()
        n, new = g.GetNumberOfSamples(), g.GetNewSamples()
        s.evaluate(g, n - new, new)
        g.ComputeErrors()
    want = a.dump_state()
    img = torch.zeros(H, W, 4, device="cuda")
    a.Integrate(img, W, H)
    for g in (b, c):
        assert_states_equal(g.dump_state(), want, keys=KEYS, what="a pass after the render")
        out = torch.zeros(H, W, 4, device="cuda")
        g.Integrate(out, W, H)
        ok, worst = rel_close(out.cpu().numpy(), img.cpu().numpy())
        assert ok, worst
        assert g.Validate()
