"""The adjoint's gradient pass goes through columns of 32 consecutive z of one |kx|, |ky|:
gradients at grids whose rows end before, at and after a column's end, with all rows that
are their own mirror image (kx or ky of 0 and N/2), against the FP64 reference adjoint.

Tolerance 1e-5 of the largest gradient, as in test_gpu_adjoint.py: a mode's cotangent is
formed in single precision from its inputs (about ten roundings of 6e-8), a bin's total
from at most 1e5 of them in sums of 32."""
import numpy as np
import pytest

from test_gpu_adjoint import gpu_grads, setup

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,nb", [(30, 20), (62, 40), (66, 90)])
def test_column_edges(gpu, oracle, N, nb):
    c, ref, k, a = setup(oracle, gpu, N, nb, 16, (0.05, 0.05, 0.05), seed=N)
    wb = np.random.default_rng(N).random(c["nk"])
    xg, Dg, mg, out, pnu = gpu_grads(k, c, a, wb, recompute=False)
    adj = ref.adjoint(c["grid"].astype(np.complex128), c["delta_tot"], np.array(c["MNu"]), wb)
    xr, Dr = adj["xbar"], adj["Dbar"]
    err = np.abs(xg - xr)
    half = N // 2
    for kx in (0, 1, half, half + 1, N - 1):
        for z in (0, min(31, half), half):
            assert err[kx, :, z].max() <= 1e-5 * np.max(np.abs(xr)), (kx, z)
    assert err.max() <= 1e-5 * np.max(np.abs(xr))
    assert np.max(np.abs(Dg - Dr)) <= 1e-5 * np.max(np.abs(Dr))
    assert abs(mg[0] / adj["mbar"][0] - 1) < 1e-5
    k.close()


@pytest.mark.parametrize("N,nb,Na", [(30, 20, 16), (66, 90, 2), (66, 90, 40)])
def test_output_beside_the_input(gpu, oracle, N, nb, Na):
    """The corrected grid written to another tensor, the history's splines completed after the
    binning pass (with two rows there are none): the same grid as in place (the ratio table
    is in single precision; P_nu's last bits follow the order of the binning pass's FP64 atomic adds), and
    the input as it was."""
    import torch
    c, ref, k, a = setup(oracle, gpu, N, nb, Na, (0.05, 0.05, 0.05), seed=N)
    g = torch.as_tensor(c["grid"]).cuda()
    g0, out, work = g.clone(), torch.full_like(g, float("nan")), g.clone()
    p1, p2 = (torch.empty(c["nk"], dtype=torch.float64, device="cuda") for _ in range(2))
    torch.cuda.synchronize()
    k.diff_forward(a, c["L"], g, out, N, p1, True)
    k.diff_forward(a, c["L"], work, work, N, p2, True)
    assert torch.equal(g, g0) and torch.equal(out, work)
    assert out[0, 0, 0] == g[0, 0, 0] and not torch.equal(out, g)
    k.close()


@pytest.mark.parametrize("N,nb", [(30, 20), (48, 500)])
@pytest.mark.parametrize("recompute", [False, True])
def test_history_gradient_of_three_mass_states(gpu, oracle, N, nb, recompute):
    """The derivatives of the integrals, made without the cotangent and summed over the species
    afterwards: a block per (species, bin) and, from 608 of them up, a warp."""
    c, ref, k, a = setup(oracle, gpu, N, nb, 16, (0.02, 0.03, 0.06), seed=N)
    assert (3 * c["nk"] >= 608) == (nb == 500)
    wb = np.random.default_rng(N).random(c["nk"])
    xg, Dg, mg, out, pnu = gpu_grads(k, c, a, wb, recompute=recompute)
    adj = ref.adjoint(c["grid"].astype(np.complex128), c["delta_tot"], np.array(c["MNu"]), wb)
    xr, Dr = adj["xbar"], adj["Dbar"]
    assert np.max(np.abs(xg - xr)) <= 1e-5 * np.max(np.abs(xr))
    assert np.max(np.abs(Dg - Dr)) <= 1e-5 * np.max(np.abs(Dr))
    for i in range(3):
        assert abs(mg[i] / adj["mbar"][i] - 1) < 1e-5
    k.close()
