"""A call's preparation (fslength table, node table, knot factorisation, row splines) where
its rules change: the quadrature rule of the fslength segments by the node spacing
h = log(a / a0) / (16 rows - 1) (5e-3: 58 rows up to a = 1; 1.5e-3: 192 rows), blocks of 57,
32 and 16 segments that end on and just past the table's end, tables shorter than one block,
and row splines of 1 to 3 unknowns.  delta_nu against the oracle within its 1e-10."""
import numpy as np
import pytest

import cases
import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,a_end", [(1, 0.0105), (2, 0.02), (3, 0.03), (4, 0.5), (57, 1.0), (58, 1.0), (59, 1.0),
                                        (191, 1.0), (192, 1.0), (193, 1.0), (228, 1.0), (229, 1.0)])
def test_update_at_rule_edges(gpu, oracle, rows, a_end):
    c = cases.make_case(32, 12, rows, a_end, (0.05, 0.1, 0.1), grid=False)
    _, s = cases.oracle_state(oracle, c)
    k = cases.gpu_instance(gpu, c)
    d = np.sqrt(W.spectrum(c["kphys"]))
    for a in (a_end + 0.002, a_end + 0.004, a_end + 0.012):
        st, ref = oracle.get_delta_nu_update(s, a, c["kphys"], d)
        assert st == 0
        got = k.get_delta_nu_update(a, c["kphys"], d)
        assert cases.rel_err(got, ref) < 1e-10, a
    k.close()
