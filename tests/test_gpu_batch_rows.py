"""The batch solves the history splines 32 rows by 32 knots at a time: instances whose bins
and history end before, at and after those, against single instances of the same inputs.

Tolerance 1e-12 relative, that of test_gpu_batch.py: both solve the same well-conditioned
system (diagonally dominant, condition number below 4) in FP64."""
import numpy as np
import pytest

import cases
from test_gpu_batch import build_instance, make_params

pytestmark = pytest.mark.gpu


def test_row_and_knot_tile_edges(gpu):
    edges = [(2, 2), (3, 31), (4, 32), (32, 33), (33, 64), (34, 65), (65, 32), (66, 33), (67, 2)]  # (rows, bins)
    ps = make_params(len(edges), seed=11)
    batch, twins = [], []
    for p, (rows, nk) in zip(ps, edges):
        p.update(Na=rows, nk=nk, k=np.geomspace(p["k"][0], p["k"][-1], nk))
        batch.append(build_instance(gpu, p)[0])
        twins.append(build_instance(gpu, p)[0])
    B = gpu.KspaceBatch(batch)
    dcdm = np.concatenate([np.linspace(1.0, 2.0, nk) for _, nk in edges])
    nks = np.array([nk for _, nk in edges], dtype=np.int32)
    a0 = max(p["a_end"] for p in ps)
    B.init(np.full(len(edges), a0), nks, np.concatenate([p["k"] for p in ps]), dcdm)
    for a in (a0, a0 + 0.004, a0 + 0.012, a0 + 0.03):  # the first call (both initialised at it), a row dropped, rows kept
        out = B.step(np.full(len(edges), a), dcdm)
        assert not B.status().any(), B.status()
        for i, t in enumerate(twins):
            s = slice(int(B.offsets[i]), int(B.offsets[i + 1]))
            ref = t.get_delta_nu_update(a, ps[i]["k"], dcdm[s])
            assert np.any(ref != 0)
            assert cases.rel_err(out[s], ref) <= 1e-12, (edges[i], a)
    B.close()
    for k in batch + twins:
        k.close()
