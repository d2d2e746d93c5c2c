"""Gradients of the priority MLP at row counts around one tile and around a whole wave of
persistent CTAs (two per SM), into buffers at 16-byte and at 4-byte alignment, against the
same arithmetic in torch (tolerance as in test_learned: a BF16 rounding of layer 1 may flip).

The two alignments add the same terms in different orders.  A gradient or the loss is the
sum of at most 4 warps x 304 CTAs partial sums (b3: 4 warps x tiles), so each result is
within terms * 2^-24 times the sum of magnitudes of the exact sum, and the two within twice
that of each other; the magnitudes are summed over the rows by torch."""
import ctypes as C

import pytest

import pmdas_gb300 as P  # noqa: F401
from pmdas_gb300 import _native as N
from tests.test_learned import (IN, OFF_B1, OFF_B2, OFF_B3, OFF_W1, OFF_W2, OFF_W3, make_params, ref_forward,
                                ref_gradients, unpack)

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m", [1, 31, 127, 128, 129, 304 * 128 - 1, 304 * 128, 304 * 128 + 1, 3 * 304 * 128 + 77])
def test_gradients_at_tile_and_wave_edges(cuda, m):
    torch = cuda
    p = make_params(torch, 11 + m)
    gen = torch.Generator().manual_seed(m)
    x = torch.randn(m, IN, generator=gen).cuda()
    y = torch.randn(m, generator=gen).cuda() * 0.3
    want, lw = ref_gradients(p, x, y)
    _, h1, z2, h2, pred = ref_forward(p, x)
    dpred = (2.0 / m) * (pred - y).abs().double()
    dz2 = dpred[:, None] * unpack(p)[4].abs().double()[None, :] * (z2 > 0)
    dz1 = (dz2 @ unpack(p)[2].abs().double()) * (h1 > 0)
    most = torch.zeros(N.MLP_PARAMS, dtype=torch.float64, device="cuda")
    most[OFF_W1:OFF_B1] = (dz1.T @ x.abs().double()).reshape(-1)
    most[OFF_B1:OFF_W2] = dz1.sum(0)
    most[OFF_W2:OFF_B2] = (dz2.T @ h1.double()).reshape(-1)
    most[OFF_B2:OFF_W3] = dz2.sum(0)
    most[OFF_W3:OFF_B3] = h2.double().T @ dpred
    most[OFF_B3] = dpred.sum()
    terms = 4 * max(304, (m + 127) // 128)
    buf = torch.full((2, N.MLP_PARAMS + 8), 7.0, device="cuda")
    got, losses = [], []
    for k, off in enumerate((4, 5)):
        loss, out = C.c_float(), buf[k, off:off + N.MLP_PARAMS]
        N.check(N.load().mdas_mlp_gradients(p.data_ptr(), x.data_ptr(), y.data_ptr(), m, out.data_ptr(),
                                            C.byref(loss), None), "gradients")
        assert (buf[k, :off] == 7.0).all() and (buf[k, off + N.MLP_PARAMS:] == 7.0).all()
        got.append(out.clone())
        losses.append(loss.value)
        assert abs(loss.value - lw) <= 1e-3 * max(abs(lw), 1e-6)
        for name, a, b in (("W1", OFF_W1, OFF_B1), ("b1", OFF_B1, OFF_W2), ("W2", OFF_W2, OFF_B2),
                           ("b2", OFF_B2, OFF_W3), ("w3", OFF_W3, OFF_B3), ("b3", OFF_B3, OFF_B3 + 1)):
            s = want[a:b].abs().max().item() + 1e-9
            assert (out[a:b] - want[a:b]).abs().max().item() / s < 5e-3, name
    assert ((got[0] - got[1]).abs().double() <= 2 * terms * 2.0 ** -24 * most + 1e-30).all()
    assert abs(losses[0] - losses[1]) <= 2 * terms * 2.0 ** -24 * losses[0]
