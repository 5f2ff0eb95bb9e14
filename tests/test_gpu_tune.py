"""Autotuned handles that share a grid.

The launch geometry is tuned once per (grid, precision, device) and read back
from the process's cache by every later handle of that grid, also where the
grid runs compile-time passes and nothing is tuned: those handles must run the
same passes as the first, so their steps are bit-identical.
"""
import numpy as np
import pytest

from ftspolysol_b200.cases import Case, homopolymer
from ftspolysol_b200.derive import derive

pytestmark = pytest.mark.gpu


def case_of(m):
    V = 0.125 * m[0] * m[1] * m[2]
    return Case(name="t", m=m, dL=0.5, monomer_names=["A"], chi=[0.0], xi=0.1, lB=1.0,
                species=[homopolymer("P", 2 * max(1, int(round(0.25 * V / 5))), 5)],
                counterions={"number": "auto_neutralize", "valence": 1.0}, dt=0.01, init_seed=4)


@pytest.mark.parametrize("m", [(32, 32, 32), (64, 64, 64), (20, 18, 15), (64, 32, 32), (128, 16, 12)], ids=lambda m: "%dx%dx%d" % m)
@pytest.mark.parametrize("prec", ["fp64", "fp32"])
def test_handles_of_one_grid(m, prec):
    from ftspolysol_b200 import Engine, FP32, FP64, SCHEME_SI
    case = case_of(m)
    d = derive(case)
    om, ps = case.initial_fields()
    out = []
    for _ in range(3):
        e = Engine(d, precision=FP64 if prec == "fp64" else FP32, scheme=SCHEME_SI, noise=True, seed=5, autotune=True)
        e.set_fields(om, ps)
        rec = e.step()[1]
        out.append((e.tune_info(), rec, e.get("omega"), e.get("psi")))
        e.close()
    assert out[1][0]["cached"] == 1 and out[2][0]["cached"] == 1
    for t, rec, w, p in out[1:]:
        assert (t["max_radix"], t["tile_width"]) == (out[0][0]["max_radix"], out[0][0]["tile_width"])
        np.testing.assert_array_equal(rec, out[0][1])
        np.testing.assert_array_equal(w, out[0][2])
        np.testing.assert_array_equal(p, out[0][3])
