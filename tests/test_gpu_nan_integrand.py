"""A NaN in one bin's history makes every error estimate of that bin's integral NaN: the search for
the largest of them still names an interval of the list, in every shape of the integral kernel
(blocks of 2, 4, 8 and 12 warps, a warp, the rounds of two intervals of hybrid neutrinos, the
batch).  The call ends in the error of a failed integral (2001) or of a NaN delta_nu (2004), as
test_gpu_errors.py has it, and the other bins are what they are without it: bit for bit, each
bin's integral being its own."""
import numpy as np
import pytest

import cases
import workloads as W

pytestmark = pytest.mark.gpu


NK, BAD = 24, 7
KK = np.geomspace(0.01, 5.0, NK)
DCDM = np.sqrt(W.spectrum(KK))


def _history(bad):
    sf, dt = W.history(KK, 30, 1.0)
    if bad:
        dt[BAD, 11] = np.nan
    return sf, dt


def _instance(gpu, hybrid):
    k = gpu.KspaceNeutrinos()
    k.init_omega_nu((0.1, 0.1, 0.1), 0.01, 0.7)
    if hybrid:
        k.init_hybrid_nu(700.0, 299792.458, 0.5)
    k.set_hubble(0.3)
    k.alloc_table(NK, 0.01, 0.5, 0.3, W.UNIT_TIME, W.UNIT_LENGTH_MPC)
    k.set_transfer(*W.transfer_table(0.3))
    k.set_nu_state(*_history(False))
    return k


def _check(k, good):
    last, ref = (x.vectors()["delta_nu_last"][:NK] for x in (k, good))
    rest = np.arange(NK) != BAD
    assert np.isnan(last[BAD]) and np.all(np.isfinite(ref)) and np.array_equal(last[rest], ref[rest])


@pytest.mark.parametrize("hybrid", [False, True])
@pytest.mark.parametrize("split", ["0", "1", "2", "4", "8", "12"])
def test_nan_history_in_every_shape(gpu, monkeypatch, hybrid, split):
    monkeypatch.setenv("KSPACE_GPU_QAG_SPLIT", split)
    k, good = _instance(gpu, hybrid), _instance(gpu, hybrid)
    for x, bad in ((k, True), (good, False)):
        x.get_delta_nu_update(1.0, KK, DCDM)
        x.set_nu_state(*_history(bad))
    good.get_delta_nu_update(1.02, KK, DCDM)
    with pytest.raises(gpu.KspaceError) as e:
        k.get_delta_nu_update(1.02, KK, DCDM)
    assert e.value.code in (2001, 2004)
    _check(k, good)
    good.close()
    k.close()


def test_nan_history_of_a_batch_member(gpu):
    ks = [_instance(gpu, False) for _ in range(2)]
    B = gpu.KspaceBatch(ks)
    a, pool = np.ones(2), np.tile(DCDM, 2)
    B.init(a, np.array([NK, NK], dtype=np.int32), np.tile(KK, 2), pool)
    B.step(a, pool)
    for x, bad in zip(ks, (True, False)):
        x.set_nu_state(*_history(bad))
    with pytest.raises(gpu.KspaceError):
        B.step(1.02 * a, pool)
    st = B.status()
    assert st[0] in (2001, 2004) and st[1] == 0
    _check(*ks)
    B.close()
    for k in ks:
        k.close()
