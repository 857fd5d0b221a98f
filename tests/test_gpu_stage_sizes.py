"""Stage kernels around the sizes where their dispatch changes, bit-identical to
the oracle: the Gram's copies go subcarrier by subcarrier above 64 pieces."""
from __future__ import annotations

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


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
