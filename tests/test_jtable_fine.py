"""The fine table of J(x) (csrc/jfine_table.h, the delta_nu integrals' own) against the
fitting formula in 40-digit arithmetic, with the piece selection of ksp_jfit.cuh: octave and
mantissa bits of x rounded to single precision, so that x may lie a single-precision rounding
outside its piece.  The first table's bound holds: 5e-16."""
import os
import struct

import numpy as np
import pytest

pytest.importorskip("mpmath")

import test_jtable as base


def test_fine_table_matches_formula(monkeypatch):
    monkeypatch.setattr(base, "HDR", os.path.join(os.path.dirname(base.HDR), "jfine_table.h"))
    text = open(base.HDR).read().replace("KSP_JFINE", "KSP_JFIT")
    monkeypatch.setattr("builtins.open", lambda *a, **k: __import__("io").StringIO(text))
    m, T = base.load()
    monkeypatch.undo()
    assert T.shape == (6400, 8) and not T[:, 7].any()
    e0, bits = m["KSP_JFIT_E0"], m["KSP_JFIT_SUB_BITS"]
    rng = np.random.default_rng(1)
    xs = list(np.exp(rng.uniform(np.log(2.0 ** e0), np.log(2.0 ** m["KSP_JFIT_E1"]) - 1e-6, 3000)))
    for e in range(e0, m["KSP_JFIT_E1"], 3):  # just below and above piece edges, to half a rounding
        for s in range(1, 256, 17):
            x = 2.0 ** e * (1 + s / 256)
            xs += [x, x * (1 - 2.0 ** -25), x * (1 - 2.0 ** -26), x * (1 + 2.0 ** -25)]
    worst = 0.0
    for x in xs:
        f = struct.unpack("<I", struct.pack("<f", np.float32(x)))[0]
        p = T[(f >> (23 - bits)) - ((127 + e0) << bits)]
        t, v = x - p[0], 0.0
        for c in reversed(p[1:7]):
            v = v * t + c
        ex = base.J_exact(x)
        worst = max(worst, abs(float((v - ex) / ex)))
    assert worst < 5e-16, worst
