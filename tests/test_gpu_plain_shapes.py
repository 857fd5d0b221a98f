"""The plain FP32 chain and its stages at the sizes where their kernel's
division of a subcarrier among lanes can go wrong: layers around each tile
(2, 4, 8, 16), odd antenna counts, antennas just past a team's lanes, one and
sixteen symbols, rows that are only 8-byte aligned, and several cells of
different shapes in one call.  Every result is bit-identical to the oracle."""
from __future__ import annotations

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

SHAPES = [  # (nPRB, nAnt, nLayers, nSym, qam)
    (1, 1, 1, 1, 4), (1, 17, 1, 16, 16), (2, 16, 2, 9, 64), (1, 33, 3, 5, 256), (3, 32, 4, 13, 16),
    (1, 20, 5, 16, 4), (1, 65, 7, 3, 64), (2, 64, 8, 14, 256), (1, 31, 8, 16, 16), (1, 129, 9, 8, 64),
    (1, 40, 12, 7, 256), (1, 127, 15, 11, 16), (1, 256, 16, 16, 256),
]


def _d(x, dev):
    return torch.from_numpy(np.ascontiguousarray(x)).to(dev)


def _shifted(x, cuda, shift):
    """x on the device, `shift` complex values past a 16-byte boundary."""
    t = torch.empty(x.numel() + 2, dtype=x.dtype, device=cuda)
    v = t[shift:shift + x.numel()]
    v.copy_(x.reshape(-1))
    return v


def _desc(aeq, c, cuda, shift, yeq=True):
    H, Y = _shifted(c.H, cuda, shift), _shifted(c.Y, cuda, shift)
    llr = torch.full((c.llr_numel,), float("nan"), dtype=torch.float32, device=cuda)
    ye = torch.full((c.nSC * c.nLayers * c.nSym,), float("nan"), dtype=torch.complex64, device=cuda) if yeq else None
    return aeq.cell_desc(H, Y, llr, c.sigma2, c.nPRB, c.nAnt, c.nLayers, c.nSym, c.nPamBits, Y_eq=ye), (H, Y, llr, ye)


def _check(orc, c, llr, ye):
    y32, _, l32 = orc.chain_f32(c.H.numpy(), c.Y.numpy(), c.sigma2, c.nSC, c.nAnt, c.nLayers, c.nSym, c.nPamBits)
    np.testing.assert_array_equal(llr.cpu().numpy(), l32)
    if ye is not None:
        np.testing.assert_array_equal(ye.cpu().numpy(), y32)


@pytest.mark.parametrize("shift", [0, 1])
@pytest.mark.parametrize("shape", SHAPES)
def test_chain_and_stages_bit_exact(aeq, wl, orc, cuda, shape, shift):
    p, A, L, S, q = shape
    c = wl.make_cell(p, A, L, S, q, 20.0, seed=100 + A)
    d, (H, Y, llr, ye) = _desc(aeq, c, cuda, shift)
    aeq.pusch_eq_plain([d], torch.empty(aeq.pusch_eq_plain_workspace([d]), dtype=torch.uint8, device=cuda))
    n = c.nSC
    G = _shifted(torch.zeros(n * L * L, dtype=torch.complex64), cuda, shift)
    C = _shifted(torch.zeros(n * L * A, dtype=torch.complex64), cuda, shift)
    ni = torch.zeros(n * L, dtype=torch.float32, device=cuda)
    O = _shifted(torch.zeros(n * L * S, dtype=torch.complex64), cuda, shift)
    aeq.gram(H, c.sigma2, G, n, A, L)
    aeq.mmse_coef(G, H, C, ni, n, A, L)
    aeq.coef_apply(C, Y, O, n, S, L, A)
    torch.cuda.synchronize()
    Gr = orc.gram(c.H.numpy(), c.sigma2, n, A, L)
    Cr, nr = orc.mmse_coef(Gr, c.H.numpy(), n, A, L)
    np.testing.assert_array_equal(G.cpu().numpy(), Gr)
    np.testing.assert_array_equal(C.cpu().numpy(), Cr)
    np.testing.assert_array_equal(ni.cpu().numpy(), nr)
    np.testing.assert_array_equal(O.cpu().numpy(), orc.coef_apply_v1(Cr, c.Y.numpy().reshape(-1), n, S, L, A))
    _check(orc, c, llr, ye)


def test_many_cells_in_one_call(aeq, wl, orc, cuda):
    """More cells than one launch holds, tiles changing from cell to cell, every other cell without Y_eq."""
    cells = [wl.make_cell(*SHAPES[i % 8], 20.0, seed=i) for i in range(12)]
    cells += [wl.make_cell(1, 8, 2, 4, 16, 20.0, seed=50 + i) for i in range(70)]
    got = [_desc(aeq, c, cuda, 0, yeq=i % 2 == 0) for i, c in enumerate(cells)]
    arr = (aeq.CellDesc * len(cells))(*[d for d, _ in got])
    ws = torch.empty(aeq.lib().aerial_pusch_eq_plain_workspace(arr, len(cells)), dtype=torch.uint8, device=cuda)
    assert aeq.lib().aerial_pusch_eq_plain(arr, len(cells), ws.data_ptr(), ws.numel(), None) == 0
    torch.cuda.synchronize()
    for c, (_, (_, _, llr, ye)) in zip(cells, got):
        _check(orc, c, llr, ye)


@pytest.mark.parametrize("n", [1, 2, 3, 4])
@pytest.mark.parametrize("N,spn,shift", [(1, 1, 0), (511, 11, 0), (513, 1, 0), (5000, 1023, 0), (5000, 1024, 0),
                                         (5000, 1025, 0), (4096, 7, 2), (1025, 14, 4)])
def test_llr_sizes_bit_exact(aeq, orc, cuda, n, N, spn, shift):
    """Partial blocks, symbols per noise value around the fast quotient's limit, outputs off the wide alignment."""
    rng = np.random.default_rng(N + n)
    soft = (rng.standard_normal(2 * N) * 0.7).astype(np.float32)
    ni = (10 ** rng.uniform(0, 3, N // spn + 1)).astype(np.float32)
    buf = torch.full((N * 2 * n + 16,), float("nan"), dtype=torch.float32, device=cuda)
    out = buf[shift:shift + N * 2 * n]
    aeq.llr_f32(_d(soft, cuda), _d(ni, cuda), out, N, n, spn)
    s16, ni1 = orc.ref_llr_inputs(N, N)
    buf16 = torch.full((N * 2 * n + 16,), -1, dtype=torch.int16, device=cuda)
    out16 = buf16[shift:shift + N * 2 * n]
    aeq.llr(_d(s16.view(np.int16), cuda), _d(ni1, cuda), out16, N, n)
    torch.cuda.synchronize()
    np.testing.assert_array_equal(out.cpu().numpy(), orc.llr_f32(soft.view(np.complex64), ni, n, spn))
    np.testing.assert_array_equal(out16.cpu().numpy().view(np.uint16), orc.llr_f16io(s16, ni1, n))
    assert torch.isnan(buf[:shift]).all() and torch.isnan(buf[shift + N * 2 * n:]).all()     # nothing else written
    assert (buf16[:shift] == -1).all() and (buf16[shift + N * 2 * n:] == -1).all()


@pytest.mark.parametrize("shift", [0, 1])
@pytest.mark.parametrize("shape", [(1, 1, 1, 1), (13, 8, 8, 8), (24, 31, 9, 9), (12, 32, 16, 16), (12, 40, 8, 14),
                                   (12, 65, 3, 11), (12, 256, 16, 7)])
def test_coef_apply_tc_sizes(aeq, orc, cuda, shape, shift):
    """Tiles with missing layers and symbols, antenna counts around the groups of four k-steps (32 antennas)."""
    nSC, A, L, S = shape
    v = orc.ref_uniform(7, nSC * L * A * 2 + nSC * S * A * 2, 1.0)
    C = v[: nSC * L * A * 2].view(np.complex64)
    Y = v[nSC * L * A * 2:].view(np.complex64)
    O = torch.zeros(nSC * L * S, dtype=torch.complex64, device=cuda)
    aeq.coef_apply_tc(_shifted(torch.from_numpy(C.copy()), cuda, shift), _shifted(torch.from_numpy(Y.copy()), cuda, shift),
                      O, nSC, S, L, A)
    torch.cuda.synchronize()
    ref = orc.coef_apply_v2_model(C, Y, nSC, S, L, A)
    # both sum the same exact FP16 products in FP32, in another order: A complex products of size <= 1/2 each
    np.testing.assert_allclose(O.cpu().numpy(), ref, rtol=0, atol=2 * A * 2.0 ** -23 * max(1.0, A / 8))
