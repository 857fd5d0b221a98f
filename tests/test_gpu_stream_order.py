"""Kernels launched to overlap the end of the previous one read what it wrote:
chains of the library's kernels and of torch's, enqueued back to back with
their intermediates overwritten in between, and captured in a graph, give the
results of the same calls with a synchronisation after each, bit for bit."""
from __future__ import annotations

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

REPS = 20


def _cplx(n, g, cuda, shift=0):
    """n complex values, `shift` values past a 16-byte boundary."""
    t = torch.empty(n + 2, dtype=torch.complex64, device=cuda)[shift:shift + n]
    t.copy_(torch.randn(n, generator=g, dtype=torch.complex64))
    return t


def _stages(aeq, cuda, A, shift):
    """Gram -> MMSE coefficients -> coef_apply on the tensor cores -> both demappers."""
    n, L, S, pam = 1584, 8, 14, 4
    g = torch.Generator().manual_seed(A + shift)
    H, Y = _cplx(n * A * L, g, cuda) * (1 / A) ** 0.5, _cplx(n * S * A, g, cuda, shift)
    G, C = _cplx(n * L * L, g, cuda), _cplx(n * L * A, g, cuda, shift)
    ni, O = torch.empty(n * L, device=cuda), _cplx(n * L * S, g, cuda)
    llr = torch.empty(n * L * S * 2 * pam, device=cuda)
    O16 = torch.empty(2 * n * L * S, dtype=torch.float16, device=cuda)
    ni16, llr16 = torch.empty(n * L * S, device=cuda), torch.empty(n * L * S * 2 * pam, dtype=torch.float16, device=cuda)
    mid = [torch.view_as_real(G), torch.view_as_real(C), ni, torch.view_as_real(O), O16, ni16]
    calls = [lambda: aeq.gram(H, 0.01, G, n, A, L), lambda: aeq.mmse_coef(G, H, C, ni, n, A, L),
             lambda: aeq.coef_apply_tc(C, Y, O, n, S, L, A), lambda: aeq.llr_f32(O, ni, llr, n * L * S, pam, S),
             lambda: O16.copy_(torch.view_as_real(O).reshape(-1)),
             lambda: ni16.view(n * L, S).copy_(ni[:, None].expand(-1, S)),
             lambda: aeq.llr(O16, ni16, llr16, n * L * S, pam)]
    return calls, mid, [llr, llr16]


def _filters(aeq, cuda, taps, shift):
    """torch's taps and pilots -> the filter -> the equalizer (and the plain chain) on the channel it wrote."""
    blocks, A, L, S, pam = 132 * 12 // taps, 64, 4, 11, 2
    g = torch.Generator().manual_seed(taps)
    src = [torch.randn(k, generator=g).to(cuda) for k in (2 * blocks * A * taps, 2 * taps * taps, 2 * L * 4)]
    P, W, F = (torch.empty(s.numel(), dtype=torch.float16, device=cuda) for s in src)
    nSC = blocks * taps
    H, Y = _cplx(nSC * A * L, g, cuda), _cplx(nSC * S * A, g, cuda, shift)
    outs = [torch.empty(nSC * L * S * 2 * pam, device=cuda) for _ in range(2)]
    d = [aeq.cell_desc(H, Y, o, 0.01, nSC // 12, A, L, S, pam) for o in outs]
    ws = torch.empty(aeq.pusch_eq_plain_workspace(d[1:]), dtype=torch.uint8, device=cuda)
    est = (lambda: aeq.srs_to_channel(H, P, W, F, A, blocks, taps, L, 4)) if taps <= 24 else (
        lambda: aeq.chest_interp(H, P, W, F, A, blocks, taps, taps, L, 4))
    calls = [lambda: [t.copy_(s * 0.1) for t, s in zip((P, W, F), src)], est, lambda: aeq.pusch_eq_fused(d[:1]),
             lambda: aeq.pusch_eq_plain(d[1:], ws)]
    return calls, [P, W, F, torch.view_as_real(H)], outs


CHAINS = {"stages": (_stages, 64, 0), "stages odd antennas": (_stages, 63, 0), "stages shifted": (_stages, 64, 1),
          "srs": (_filters, 12, 0), "srs shifted": (_filters, 24, 1), "chest": (_filters, 96, 0)}


@pytest.mark.parametrize("captured", [False, True], ids=["stream", "graph"])
@pytest.mark.parametrize("name", CHAINS)
def test_back_to_back_equals_synchronised(aeq, cuda, name, captured):
    make, a, shift = CHAINS[name]
    calls, mid, outs = make(aeq, cuda, a, shift)
    for c in calls:
        c()
        torch.cuda.synchronize()
    ref = [o.cpu().numpy().copy() for o in outs]
    assert all(np.isfinite(r).all() for r in ref)

    def chain():
        for t in mid + outs:
            t.fill_(float("nan"))
        for c in calls:
            c()

    stream = torch.cuda.Stream()
    got = []
    with torch.cuda.stream(stream):
        if captured:
            graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(graph, stream=stream):
                chain()
        for _ in range(REPS):
            graph.replay() if captured else chain()
            got.append([o.clone() for o in outs])
    torch.cuda.synchronize()
    for run in got:
        for r, o in zip(ref, run):
            np.testing.assert_array_equal(o.cpu().numpy(), r)
