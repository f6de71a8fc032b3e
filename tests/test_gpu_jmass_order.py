"""set_jmass is complete when it returns, whatever its context's stream is busy with: a batch that
reads the masses on its own streams, and a context whose stream is changed, use the new ones.

Tolerance 1e-12 relative, that of test_gpu_batch.py for a member against a single instance."""
import numpy as np
import pytest

import cases
import workloads as W

pytestmark = pytest.mark.gpu
OLD, NEW = (0.02, 0.03, 0.06), (0.05, 0.08, 0.11)


def _busy(torch):
    """A stream with a tenth of a second of work on it."""
    s = torch.cuda.Stream()
    with torch.cuda.stream(s):
        torch.cuda._sleep(200_000_000)
    return s


def _start(gpu, c, dcdm):
    k = cases.gpu_instance(gpu, c)
    k.get_delta_nu_update(0.51, c["kphys"], dcdm)
    return k


@pytest.mark.parametrize("graph", [False, True])
def test_batch_step_after_set_jmass(gpu, graph):
    import torch
    c = cases.make_case(32, 32, 10, 0.5, OLD, grid=False)
    dcdm = np.sqrt(W.spectrum(c["kphys"]))
    nk = np.array([c["nk"]], dtype=np.int32)
    k, twin, old = cases.gpu_instance(gpu, c), _start(gpu, c, dcdm), _start(gpu, c, dcdm)
    B = gpu.KspaceBatch([k])
    B.set_tuning(use_graph=graph)
    B.init(np.array([0.51]), nk, c["kphys"], dcdm)
    for a in (0.51, 0.515):  # with a graph, the second step is the captured one
        B.step(np.array([a]), dcdm)
    for x in (twin, old):
        x.get_delta_nu_update(0.515, c["kphys"], dcdm)
    twin.set_jmass(NEW)
    want, before = (x.get_delta_nu_update(0.53, c["kphys"], dcdm) for x in (twin, old))
    assert cases.rel_err(want, before) > 1e-3
    s = _busy(torch)
    k.set_stream(s.cuda_stream)
    k.set_jmass(NEW)
    got = B.step(np.array([0.53]), dcdm)
    assert cases.rel_err(got, want) <= 1e-12
    torch.cuda.synchronize()
    k.set_stream(0)
    B.close()
    for x in (k, twin, old):
        x.close()


def test_stream_changed_after_set_jmass(gpu):
    import torch
    c = cases.make_case(32, 32, 10, 0.5, OLD, grid=False)
    dcdm = np.sqrt(W.spectrum(c["kphys"]))
    k = _start(gpu, c, dcdm)
    s = _busy(torch)
    k.set_stream(s.cuda_stream)
    k.set_jmass(NEW)
    assert s.query()  # nothing of the call is left on the stream it was made on
    k.set_stream(0)
    twin = _start(gpu, c, dcdm)
    twin.set_jmass(NEW)
    assert cases.rel_err(k.get_delta_nu_update(0.53, c["kphys"], dcdm),
                         twin.get_delta_nu_update(0.53, c["kphys"], dcdm)) <= 1e-12
    k.close()
    twin.close()
