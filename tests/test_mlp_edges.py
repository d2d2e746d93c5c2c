"""Gradients of the priority MLP into a buffer at 16-byte and at 4-byte alignment
(vector and scalar additions), at row counts around one tile and around a whole
wave of persistent CTAs (two per SM).  The two results add the same per-CTA
partial sums in different orders: at most 304 of them, so 304 * 2^-24 of the
largest sum of magnitudes, taken as 64 times the largest gradient, bounds the
difference."""
import ctypes as C

import pytest

from pmdas_gb300 import _native as N

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m", [1, 127, 128, 129, 2 * 152 * 128, 2 * 152 * 128 + 1])
def test_gradients_at_both_alignments(cuda, m):
    torch = cuda
    gen = torch.Generator().manual_seed(m)
    p = ((torch.rand(N.MLP_PARAMS, generator=gen) * 2 - 1) * 0.2).cuda()
    x = torch.randn(m, 16, generator=gen).cuda()
    y = (torch.randn(m, generator=gen) * 0.1).cuda()
    buf = torch.full((2, N.MLP_PARAMS + 8), 7.0, device="cuda")
    got, losses = [], []
    for k, off in enumerate((4, 5)):
        loss = C.c_float()
        out = buf[k, off:off + N.MLP_PARAMS]
        N.check(N.load().mdas_mlp_gradients(p.data_ptr(), x.data_ptr(), y.data_ptr(), m, out.data_ptr(),
                                            C.byref(loss), None), "gradients")
        assert (buf[k, :off] == 7.0).all() and (buf[k, off + N.MLP_PARAMS:] == 7.0).all()
        got.append(out.clone())
        losses.append(loss.value)
    bound = 304 * 2.0 ** -24 * 64 * got[0].abs().max().item()
    assert (got[0] - got[1]).abs().max().item() <= bound
    assert abs(losses[0] - losses[1]) <= 304 * 2.0 ** -24 * losses[0]
