"""Compile-time plans of the split-y passes on grids that are no cubes: the
square planes of the production cubes with other x extents (one row, odd,
large), the x extents 32, 64 and 128 with rows of 4 and 8 and whole tiles of
columns, and their neighbours that must take the run-time plans (m3 no
multiple of 4, rows of 6); x extents so long that the tiles of the k-space pass
get narrower; x extents with two radices above 16 or one of 27.

Chain propagation against numpy FFTs (complex128, 1e-12 of the field's largest
modulus), densities and record of an asymmetric chain (both sweeps, stress
sums) against the oracle (1e-10; complex64: 1e-5 on fields, 2e-3 on records):
the tolerances of test_gpu_split.py.
"""
import numpy as np
import pytest

import pyoracle as po
from ftspolysol_b200.cases import Case, homopolymer
from ftspolysol_b200.derive import derive
from test_gpu_split import diblock, reference_chain

pytestmark = pytest.mark.gpu

CHAINS = [(64, 32, 32), (128, 32, 32), (1, 32, 32), (45, 32, 32), (256, 32, 32), (32, 64, 64), (125, 64, 64), (128, 64, 64),
          (10, 48, 48), (27, 96, 96), (2, 128, 128), (64, 128, 128), (32, 20, 12), (64, 16, 4), (128, 24, 20), (32, 80, 8),
          (64, 40, 36), (128, 72, 12), (32, 20, 15), (64, 48, 20), (128, 36, 8), (512, 32, 32), (512, 30, 8), (480, 64, 6), (400, 120, 4),
          (243, 32, 32), (324, 48, 48), (486, 32, 32), (500, 32, 32), (576, 32, 32), (625, 32, 32), (640, 32, 32), (729, 32, 32),
          (800, 32, 32)]


@pytest.mark.parametrize("m", CHAINS, ids=lambda m: "%dx%dx%d" % m)
def test_chain(m):
    import torch
    from ftspolysol_b200 import Engine
    case = Case(name="chain", m=m, dL=0.5, species=[homopolymer("P", 4, 4, charge=0.0)], lB=0.0, ions_enabled=False)
    rng = np.random.default_rng(9)
    w = (0.3 * rng.standard_normal(m) + 0.2j * rng.standard_normal(m)).astype(np.complex128)
    wd = torch.from_numpy(w.reshape(-1)).cuda()
    q = torch.zeros_like(wd)
    with Engine(derive(case)) as eng:
        Q = eng.propagate_chain(wd.data_ptr(), 4, 1.1, q.data_ptr())
    ref = reference_chain(w, case.L, 4, 1.1)
    assert np.max(np.abs(q.cpu().numpy().reshape(m) - ref)) / np.max(np.abs(ref)) < 1e-12
    assert abs(Q - ref.mean()) / abs(ref.mean()) < 1e-12


@pytest.mark.parametrize("m", [(64, 32, 32), (32, 64, 64), (20, 64, 64), (128, 16, 12), (128, 72, 72), (3, 128, 128), (5, 96, 96), (512, 30, 8), (243, 32, 32),
                               (640, 32, 32)],
                         ids=lambda m: "%dx%dx%d" % m)
@pytest.mark.parametrize("prec", ["fp64", "fp32"])
def test_both_sweeps(m, prec):
    from ftspolysol_b200 import Engine, FP32, FP64
    case = diblock(m)
    d = derive(case)
    om, ps = case.initial_fields()
    o = po.Oracle(d)
    o.set_fields(om, ps)
    Q = o.compute_densities(0)
    rho = o.get("rho_type")
    rec = o.measure(0, Q)
    o.close()
    ftol, rtol = (1e-10, 1e-10) if prec == "fp64" else (1e-5, 2e-3)
    with Engine(d, precision=FP64 if prec == "fp64" else FP32) as eng:
        eng.set_fields(om, ps)
        got = eng.measure(0)
        assert np.max(np.abs(eng.get("rho_type") - rho)) / np.max(np.abs(rho)) < ftol
        assert np.max(np.abs(got - rec) / np.maximum(np.abs(rec), 1e-3)) < rtol
