"""Stage kernels around the sizes where their dispatch changes, bit-identical to
the oracle: the demapper's four symbols a thread begin at a block per SM, the
Gram's copies go subcarrier by subcarrier above 64 pieces.  The tensor-core
coef_apply, within its rounding of the oracle, loads one k-step (8 antennas) or
eight at a time."""
from __future__ import annotations

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 3, 4])
@pytest.mark.parametrize("extra,spn,shift", [(-1, 14, 0), (0, 1, 0), (1, 11, 2), (255, 14, 4), (1030, 2000, 6)])
def test_demapper_around_a_block_per_sm(aeq, orc, cuda, n, extra, spn, shift):
    N = 1024 * (torch.cuda.get_device_properties(0).multi_processor_count - 1) + 1 + extra
    rng = np.random.default_rng(N + n)
    soft = (rng.standard_normal(2 * N) * 0.7).astype(np.float32)
    ni = (10 ** rng.uniform(0, 3, N // spn + 1)).astype(np.float32)
    size = N * 2 * n
    buf = torch.full((size + 16,), float("nan"), device=cuda)
    s16, ni1 = orc.ref_llr_inputs(N, N)
    buf16 = torch.full((size + 16,), -1, dtype=torch.int16, device=cuda)
    aeq.llr_f32(torch.from_numpy(soft).to(cuda), torch.from_numpy(ni).to(cuda), buf[shift:shift + size], N, n, spn)
    aeq.llr(torch.from_numpy(s16.view(np.int16)).to(cuda), torch.from_numpy(ni1).to(cuda), buf16[shift:shift + size],
            N, n)
    torch.cuda.synchronize()
    np.testing.assert_array_equal(buf[shift:shift + size].cpu().numpy(), orc.llr_f32(soft.view(np.complex64), ni, n, spn))
    np.testing.assert_array_equal(buf16[shift:shift + size].cpu().numpy().view(np.uint16), orc.llr_f16io(s16, ni1, n))
    for b, empty in ((buf, torch.isnan), (buf16, lambda t: t == -1)):              # nothing else written
        assert empty(b[:shift]).all() and empty(b[shift + size:]).all()


@pytest.mark.parametrize("shift", [0, 1])
@pytest.mark.parametrize("ant,lay", [(2, 2), (127, 1), (128, 1), (129, 1), (128, 2), (130, 2), (42, 3), (43, 3),
                                     (64, 4), (66, 4), (25, 5), (32, 8), (34, 8), (15, 16), (16, 16), (256, 2)])
def test_gram_around_the_flat_copies(aeq, wl, orc, cuda, ant, lay, shift):
    for prb in (1, 3):                                    # 12 and 36 subcarriers: warps with some missing
        c = wl.make_cell(prb, ant, min(lay, ant), 1, 4, 20.0, seed=ant + lay)
        n = c.nSC
        H = torch.empty(n * ant * lay + 2, dtype=torch.complex64, device=cuda)[shift:shift + n * ant * lay]
        if lay > ant:                                     # more layers than antennas: any values will do
            vals = torch.from_numpy(orc.ref_uniform(7, 2 * n * ant * lay, 1.0).view(np.complex64).copy())
        else:
            vals = c.H.reshape(-1)
        H.copy_(vals)
        buf = torch.full((2 * (n * lay * lay + 4),), float("nan"), device=cuda)
        G = torch.view_as_complex(buf.view(-1, 2))[shift:shift + n * lay * lay]
        aeq.gram(H, 0.25, G, n, ant, lay)
        torch.cuda.synchronize()
        np.testing.assert_array_equal(G.cpu().numpy(), orc.gram(vals.numpy(), 0.25, n, ant, lay))
        assert torch.isnan(buf[:2 * shift]).all() and torch.isnan(buf[2 * (shift + n * lay * lay):]).all()


@pytest.mark.parametrize("shift", [0, 1])
@pytest.mark.parametrize("ant", [2, 7, 8, 9, 16, 63, 64, 65, 72, 128, 130])
def test_coef_apply_tc_around_its_k_steps(aeq, orc, cuda, ant, shift):
    n, L, S = 13, 9, 9
    v = orc.ref_uniform(7, n * ant * 2 * (L + S), 1.0)
    C, Y = v[: n * L * ant * 2].view(np.complex64), v[n * L * ant * 2:].view(np.complex64)
    dev = []
    for x in (C, Y):
        t = torch.empty(x.size + 2, dtype=torch.complex64, device=cuda)[shift:shift + x.size]
        t.copy_(torch.from_numpy(x.copy()))
        dev.append(t)
    O = torch.full((n * L * S,), float("nan"), dtype=torch.complex64, device=cuda)
    aeq.coef_apply_tc(dev[0], dev[1], O, n, S, L, ant)
    torch.cuda.synchronize()
    # both sum the same exact FP16 products in FP32, in another order: ant complex products of size <= 1/2 each
    np.testing.assert_allclose(O.cpu().numpy(), orc.coef_apply_v2_model(C, Y, n, S, L, ant), rtol=0,
                               atol=2 * ant * 2.0 ** -23 * max(1.0, ant / 8))
