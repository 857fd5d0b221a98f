"""The plain chain's cells run in order and stage by stage as far as their
buffers can tell: cells that share buffers, and outputs that lie over inputs
already read, give the oracle's results bit for bit."""
from __future__ import annotations

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _oracle(orc, H, Y, c):
    y, _, l = orc.chain_f32(H, Y, c.sigma2, c.nSC, c.nAnt, c.nLayers, c.nSym, c.nPamBits)
    return l, y


def _run(aeq, descs, cuda, static=False):
    if static:
        aeq.pusch_eq_plain_static(descs)
    else:
        ws = torch.full((aeq.pusch_eq_plain_workspace(descs),), 255, dtype=torch.uint8, device=cuda)
        aeq.pusch_eq_plain(descs, ws)
    torch.cuda.synchronize()


def _desc(aeq, c, H, Y, llr, yeq=None):
    return aeq.cell_desc(H, Y, llr, c.sigma2, c.nPRB, c.nAnt, c.nLayers, c.nSym, c.nPamBits, Y_eq=yeq)


@pytest.mark.parametrize("static", [False, True])
def test_cells_sharing_buffers_run_in_order(aeq, wl, orc, cuda, static):
    """One Y_eq for all cells holds the last one's; LLRs go over the inputs of the cell before; a cell's H and Y_rx
    are what the two before it equalized (both as [subcarrier][16][16])."""
    cells = [wl.make_cell(30, 16, 16, 16, 16, 20.0, seed=900 + i) for i in range(5)]
    H, Y = [c.H.to(cuda) for c in cells], [c.Y.to(cuda) for c in cells]
    n = cells[0].nSC * 256
    shared, h4, y4 = (torch.empty(n, dtype=torch.complex64, device=cuda) for _ in range(3))
    own = [torch.empty(c.llr_numel, device=cuda) for c in cells]
    over = torch.view_as_real(H[0]).reshape(-1)                      # cell 1's LLRs: twice H[0] in size
    big = torch.empty(2 * over.numel(), device=cuda)
    big[:over.numel()].copy_(over)
    H[0] = torch.view_as_complex(big[:over.numel()].view(-1, 2))
    descs = [_desc(aeq, cells[0], H[0], Y[0], own[0], shared), _desc(aeq, cells[1], H[1], Y[1], big, shared),
             _desc(aeq, cells[2], H[2], Y[2], own[2], h4), _desc(aeq, cells[3], H[3], Y[3], own[3], y4),
             _desc(aeq, cells[4], h4, y4, own[4], shared)]
    _run(aeq, descs, cuda, static)
    ref = [_oracle(orc, c.H.numpy(), c.Y.numpy(), c) for c in cells[:4]]
    ref.append(_oracle(orc, ref[2][1], ref[3][1], cells[4]))
    for got, want in zip((own[0], big, own[2], own[3], own[4]), ref):
        np.testing.assert_array_equal(got.cpu().numpy(), want[0])
    np.testing.assert_array_equal(shared.cpu().numpy(), ref[4][1])


@pytest.mark.parametrize("static", [False, True])
@pytest.mark.parametrize("over", ["llr over H", "llr over Y", "yeq over H"])
def test_outputs_over_inputs(aeq, wl, orc, cuda, over, static):
    c, other = wl.make_cell(106, 64, 8, 11, 16, 20.0, seed=910), wl.make_cell(51, 64, 8, 11, 16, 20.0, seed=911)
    H, Y, Ho, Yo = c.H.to(cuda), c.Y.to(cuda), other.H.to(cuda), other.Y.to(cuda)
    llr, lo = torch.empty(c.llr_numel, device=cuda), torch.empty(other.llr_numel, device=cuda)
    yeq = torch.empty(c.nSC * c.nLayers * c.nSym, dtype=torch.complex64, device=cuda)
    at = torch.view_as_real(Y if over == "llr over Y" else H).reshape(-1)[256:]      # 256 values into the input
    if over.startswith("llr"):
        llr = at[:llr.numel()]
    else:
        yeq = torch.view_as_complex(at[:2 * yeq.numel()].view(-1, 2))
    descs = [_desc(aeq, other, Ho, Yo, lo), _desc(aeq, c, H, Y, llr, yeq)]
    _run(aeq, descs, cuda, static)
    l, y = _oracle(orc, c.H.numpy(), c.Y.numpy(), c)
    np.testing.assert_array_equal(llr.cpu().numpy(), l)
    np.testing.assert_array_equal(yeq.cpu().numpy(), y)
    np.testing.assert_array_equal(lo.cpu().numpy(), _oracle(orc, other.H.numpy(), other.Y.numpy(), other)[0])


def test_static_calls_overlap(aeq, wl, orc, cuda):
    """Calls on two streams at a time share nothing; each gives the oracle's results."""
    cells = [wl.make_cell(132, 64, 8, 11, 256, 25.0, seed=920), wl.make_cell(51, 32, 3, 7, 16, 20.0, seed=921)]
    ref = [_oracle(orc, c.H.numpy(), c.Y.numpy(), c) for c in cells]
    streams = [torch.cuda.Stream() for _ in cells]
    runs = []
    for c in cells:
        H, Y = c.H.to(cuda), c.Y.to(cuda)
        n = c.nSC * c.nLayers * c.nSym
        outs = [(torch.full((c.llr_numel,), float("nan"), device=cuda),
                 torch.full((n,), float("nan"), dtype=torch.complex64, device=cuda)) for _ in range(6)]
        runs.append([(o, _desc(aeq, c, H, Y, *o)) for o in outs])
    torch.cuda.synchronize()
    for step in zip(*runs):
        for (_, d), s in zip(step, streams):
            aeq.pusch_eq_plain_static([d], s)
    torch.cuda.synchronize()
    for (l, y), calls in zip(ref, runs):
        for (llr, yeq), _ in calls:
            np.testing.assert_array_equal(llr.cpu().numpy(), l)
            np.testing.assert_array_equal(yeq.cpu().numpy(), y)
