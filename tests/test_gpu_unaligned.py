"""Mixed batches whose channel or received samples start 8 bytes past a 16-byte
boundary (8-byte copies, rows padded or not), and batches in which some
subcarriers hold values that are not finite."""
from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu

ANTS, LAYERS = (16, 20, 33, 40), (1, 2, 3, 4, 8, 12, 16)


def _at(x, cuda, shift):
    """x on the device, `shift` complex values past a 16-byte boundary."""
    t = torch.empty(x.numel() + 2, dtype=torch.complex64, device=cuda)[shift:shift + x.numel()]
    t.copy_(x.reshape(-1))
    return t


def _run(aeq, cells, cuda, prec, hs=0, ys=0, spoil=None):
    descs, outs, keep = [], [], []
    for i, c in enumerate(cells):
        H, Y = _at(c.H, cuda, hs), _at(c.Y, cuda, ys)
        if spoil:
            spoil(i, c, H.view(c.nSC, -1), Y.view(c.nSC, -1))
        llr = torch.full((c.nSC, c.nLayers * c.nSym * 2 * c.nPamBits), float("nan"), device=cuda)
        yeq = torch.full((c.nSC, c.nLayers * c.nSym), float("nan"), dtype=torch.complex64, device=cuda)
        keep += [H, Y]
        outs.append((llr, torch.view_as_real(yeq)))
        descs.append(aeq.cell_desc(H, Y, llr, c.sigma2, c.nPRB, c.nAnt, c.nLayers, c.nSym, c.nPamBits, Y_eq=yeq))
    aeq.pusch_eq_fused(descs, aeq.make_tuning(prec))
    torch.cuda.synchronize()
    return outs


def _cells(wl):
    shapes = [(a, l) for a in ANTS for l in LAYERS if l <= a]
    return [wl.make_cell(1 + i % 3, a, l, (14, 7, 16, 1)[i % 4], (256, 16, 64, 4)[i % 4], 20.0, seed=300 + i)
            for i, (a, l) in enumerate(shapes)]


@pytest.mark.parametrize("prec", ["fp16", "bf16x3"])
@pytest.mark.parametrize("hs,ys", [(1, 0), (0, 1), (1, 1)])
def test_unaligned_rows_equal_aligned(aeq, wl, cuda, prec, hs, ys):
    """The same samples and the same order of every sum, so the same bits."""
    cells = _cells(wl)
    for ref, got in zip(_run(aeq, cells, cuda, prec), _run(aeq, cells, cuda, prec, hs, ys)):
        for r, g in zip(ref, got):
            assert torch.isfinite(r).all() and torch.equal(r, g)


@pytest.mark.parametrize("prec", ["fp16", "bf16x3"])
@pytest.mark.parametrize("shift", [0, 1])
def test_values_that_are_not_finite_stay_in_their_subcarrier(aeq, wl, cuda, prec, shift):
    """Unused layers and antennas of a tile are not masked: what lies in them must reach no other subcarrier."""
    cells = _cells(wl)

    def spoil(i, c, H, Y):
        if i % 3 == 2:                                  # every third cell stays clean
            return
        H[::5] = float("inf") if i % 3 else float("nan")
        Y[::4] = float("nan") if i % 3 else float("inf")

    ref = _run(aeq, cells, cuda, prec, shift, shift)
    got = _run(aeq, cells, cuda, prec, shift, shift, spoil)
    for i, (c, r, g) in enumerate(zip(cells, ref, got)):
        sc = torch.arange(c.nSC, device=cuda)
        clean = torch.ones_like(sc, dtype=torch.bool) if i % 3 == 2 else (sc % 5 != 0) & (sc % 4 != 0)
        for a, b in zip(r, g):
            assert torch.equal(a[clean], b[clean]), (i, c.nAnt, c.nLayers)
