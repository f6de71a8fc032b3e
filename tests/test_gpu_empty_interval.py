"""Calls whose integral has nothing under it: at the transfer function's scale factor a0 the
interval is empty, before it fslength is zero.  What is left is the initial-condition term, which
is delta_nu_init itself there (J(0) = 1, fslength 0), whatever an earlier call left in the tables;
an end that is no number is refused with QAG's error, and the instance stays usable.

Tolerance 1e-14: the species' weights, their sum and the products are about ten roundings."""
import math

import numpy as np
import pytest

import cases
import workloads as W

pytestmark = pytest.mark.gpu
A0 = 0.01
TOL = 1e-14


@pytest.mark.parametrize("nb,masses,split", [(24, (0.1, 0.1, 0.1), "0"), (160, (0.02, 0.03, 0.06), "0"),
                                             (500, (0.02, 0.03, 0.06), "0"), (24, (0.1, 0.1, 0.1), "1")])
def test_stored_rows_at_and_before_a0(gpu, monkeypatch, nb, masses, split):
    monkeypatch.setenv("KSPACE_GPU_QAG_SPLIT", split)
    c = cases.make_case(48, nb, 20, 0.5, masses, grid=False)
    k = cases.gpu_instance(gpu, c)
    k.delta_tot_init(c["kphys"], np.sqrt(W.spectrum(c["kphys"])), 0.51)
    nu_init = k.vectors()["delta_nu_init"][:c["nk"]]
    later = k.get_delta_nu_combined(0.4, c["kphys"])  # fills the tables
    assert cases.rel_err(later, nu_init) > 0.1
    for a in (A0, 0.9 * A0):
        assert cases.rel_err(k.get_delta_nu_combined(a, c["kphys"]), nu_init) <= TOL
        assert cases.rel_err(k.get_delta_nu(a, c["kphys"], masses[0]), nu_init) <= TOL
    for a in (math.nan, 0.0, math.inf):
        for call in (lambda: k.get_delta_nu(a, c["kphys"], masses[0]), lambda: k.get_delta_nu_combined(a, c["kphys"])):
            with pytest.raises(gpu.KspaceError) as e:
                call()
            assert e.value.code == 2001
    assert cases.rel_err(k.get_delta_nu_combined(0.4, c["kphys"]), later) <= TOL
    k.close()


def test_update_and_batch_at_a0(gpu):
    """Rows from before a0, and a call at a0: a single instance and a batch member."""
    c = cases.make_case(32, 32, 2, 0.5, (0.02, 0.03, 0.06), grid=False)
    c["scalefact"] = np.log([0.004, 0.006])
    dcdm = np.sqrt(W.spectrum(c["kphys"]))
    single, member = cases.gpu_instance(gpu, c), cases.gpu_instance(gpu, c)
    d = single.get_delta_nu_update(A0, c["kphys"], dcdm)
    nu_init = single.vectors()["delta_nu_init"][:c["nk"]]
    assert np.all(nu_init > 0) and cases.rel_err(d, nu_init) <= TOL
    B = gpu.KspaceBatch([member])
    B.init(np.array([A0]), np.array([c["nk"]], dtype=np.int32), c["kphys"], dcdm)
    assert cases.rel_err(B.step(np.array([A0]), dcdm), nu_init) <= TOL
    assert not B.status().any()
    B.close()
    single.close()
    member.close()
