"""A prepared step's provisional row is completed inside the integral kernel, whatever its shape:
a warp per integral (the default from 608 on), blocks of 2, 4, 8 and 12 warps.  Steps of the same
instance in every shape: delta_nu / delta_cdm within 1e-12 relative (the shapes take the same
decisions and differ by the rounding of sums of 61 terms) and the same subdivisions."""
import numpy as np
import pytest

import cases

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nb,Na", [(500, 20), (500, 2), (24, 33)])
def test_prepared_step_in_every_shape(gpu, monkeypatch, nb, Na):
    import torch
    c = cases.make_case(48, nb, Na, 0.5, (0.02, 0.03, 0.06), seed=nb)
    assert (3 * c["nk"] >= 608) == (nb == 500)
    ref = None
    for split in ("0", "1", "2", "4", "8", "12"):
        monkeypatch.setenv("KSPACE_GPU_QAG_SPLIT", split)
        k = cases.gpu_instance(gpu, c)
        g = torch.as_tensor(c["grid"]).cuda()
        out = []
        for a in (0.5, 0.504, 0.512, 0.53):  # the first call, a row dropped, rows kept
            torch.cuda.synchronize()
            k.add_nu_power_to_rhogrid(a, c["L"], g, 48)
            r = k.last_correction()
            out.append((r["ratio"].copy(), r["dcdm"].copy(), k.qag_stats()))
        k.close()
        if ref is None:
            ref = out
            assert any(s[1] > 0 for _, _, s in out)
        for (r, d, s), (r0, d0, s0) in zip(out, ref):
            assert s == s0, (split, s, s0)
            assert cases.rel_err(r, r0) <= 1e-12 and cases.rel_err(d, d0) <= 1e-6, split
