"""The adjoint's pass over the grid with more bins than a block of eight warps has shared memory for
(its totals take a float per bin and warp, two more per bin hold the table): fewer warps then.
384^3 in 13000 bins, 5966 of them not empty.  Against the pass that takes grids which do not lie on
16 bytes, whose totals are in FP64, for the same grid 8 bytes further on.

Tolerance 2e-5 of the largest gradient: each of the two passes is within 1e-5 of the FP64
reference (test_gpu_adjoint.py)."""
import numpy as np
import pytest

import cases
import workloads as W

pytestmark = pytest.mark.gpu


def test_more_bins_than_eight_warps_hold(gpu):
    import torch
    N, nb = 384, 13000
    c = cases.make_case(N, nb, 12, 0.5, (0.1, 0.1, 0.1), grid=False)
    nk, shape = c["nk"], (N, N, N // 2 + 1)
    assert 4 * nk * 10 > 227 * 1024 >= 4 * nk * 9
    k = cases.gpu_instance(gpu, c)
    k.delta_tot_init(c["kphys"], np.sqrt(W.spectrum(c["kphys"])), 0.51)
    grid = W.make_grid_torch(N, c["L"], seed=3)
    zero = torch.zeros(nk, dtype=torch.float64, device="cuda")  # delta_nu's cotangent from the pass alone
    got = []
    for shift in (0, 1):
        x, out, gin = (torch.zeros(grid.numel() + 2, dtype=torch.complex64, device="cuda")[shift:shift + grid.numel()]
                       .view(shape) for _ in range(3))
        x.copy_(grid)
        assert (x.data_ptr() % 16 != 0) == (shift == 1)
        pnu = torch.empty(nk, dtype=torch.float64, device="cuda")
        Dbar = torch.zeros(c["delta_tot"].shape, dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        k.diff_forward(0.51, c["L"], x, out, N, pnu, True)
        m = k.diff_backward(out, x, zero, gin, Dbar)
        got.append((gin.clone(), Dbar, torch.as_tensor(m[:1])))
    for a, b in zip(*got):
        assert b.abs().max() > 0
        assert (a - b).abs().max() <= 2e-5 * b.abs().max()
    k.close()
