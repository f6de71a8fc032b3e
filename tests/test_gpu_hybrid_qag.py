"""Hybrid neutrinos after the switch to particles: a call takes the node table of all shallow
intervals and evaluates two intervals a round (by the list of errors); a warp per integral
(KSPACE_GPU_QAG_SPLIT=1) takes one after the other from the same table, and without a node
table (KSPACE_GPU_NC_LEVELS=0) every node is evaluated where it is needed.  Same subdivisions, and
results within 1e-12 relative: the sums are of values of either sign, a few roundings of 2e-16
each, of at most 20 times their total."""
import numpy as np
import pytest

import cases
import workloads as W

pytestmark = pytest.mark.gpu


def _run(gpu, rows, nk, monkeypatch, **env):
    for name in ("KSPACE_GPU_QAG_SPLIT", "KSPACE_GPU_NC_LEVELS"):
        monkeypatch.delenv(name, raising=False)
    for name, value in env.items():
        monkeypatch.setenv(name, value)
    k = gpu.KspaceNeutrinos()
    k.init_omega_nu((0.1, 0.1, 0.1), 0.01, 0.7)
    k.init_hybrid_nu(700.0, 299792.458, 0.5)
    k.set_hubble(0.3)
    k.alloc_table(nk, 0.01, 0.01 + (rows + 20) / 100.0, 0.3, W.UNIT_TIME, W.UNIT_LENGTH_MPC)
    k.set_transfer(*W.transfer_table(0.3))
    kk = np.geomspace(0.01, 5.0, nk)
    k.set_nu_state(*W.history(kk, rows, 1.0))
    out = []
    for a in (1.0, 1.004, 1.013):
        out.append((k.get_delta_nu_update(a, kk, np.sqrt(W.spectrum(kk))), k.qag_stats()))
    k.close()
    return out


@pytest.mark.parametrize("rows,nk", [(100, 40), (30, 170)])
def test_rounds_of_two_intervals(gpu, monkeypatch, rows, nk):
    got = _run(gpu, rows, nk, monkeypatch)
    assert max(s[0] for _, s in got) > 8  # oscillating: many bisections
    for env in (dict(KSPACE_GPU_QAG_SPLIT="1"), dict(KSPACE_GPU_NC_LEVELS="0")):
        ref = _run(gpu, rows, nk, monkeypatch, **env)
        for (a, sa), (b, sb) in zip(got, ref):
            assert sa == sb, (env, sa, sb)
            assert cases.rel_err(a, b) <= 1e-12, (env, cases.rel_err(a, b))
