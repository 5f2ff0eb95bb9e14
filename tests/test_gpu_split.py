"""The split-y passes of the chain sweeps (split_passes.cuh) at the edges of
their plans: every radix, single-radix lengths, extents with a radix of 25 or
two large ones, columns that do not fill the last tile (odd m3), several row
groups per block, tiny grids, a grid that has no plan, and the production
cubes.

The chain propagation is compared with numpy FFTs (complex128, 1e-12 of the
field's largest modulus, the tolerance of the other chain tests), densities
and record of an asymmetric chain (both sweeps, stress sums) with the oracle
(1e-10; complex64: 1e-5 on fields, 2e-3 on records, as elsewhere).
"""
import numpy as np
import pytest

import pyoracle as po
from ftspolysol_b200.cases import Case, Species, homopolymer
from ftspolysol_b200.derive import derive

pytestmark = pytest.mark.gpu

CHAINS = [(2, 3, 5), (1, 4, 1), (8, 9, 10), (12, 15, 16), (18, 20, 27), (25, 30, 45), (81, 6, 75), (90, 40, 36),
          (125, 6, 8), (8, 125, 6), (6, 8, 125), (25, 125, 20), (150, 10, 12), (12, 144, 10), (10, 12, 160), (192, 6, 5),
          (4, 256, 9), (5, 6, 225), (200, 9, 4), (162, 4, 6), (6, 200, 5), (320, 8, 3), (4, 10, 384), (16, 12, 512), (243, 4, 6), (32, 32, 32), (48, 48, 48), (64, 64, 64), (96, 96, 96), (128, 128, 128)]


def reference_chain(w, L, N, b):
    k = [2 * np.pi * np.fft.fftfreq(n, d=l / n) for n, l in zip(w.shape, L)]
    k2 = k[0][:, None, None] ** 2 + k[1][None, :, None] ** 2 + k[2][None, None, :] ** 2
    e = np.exp(-w)
    q = e.copy()
    for _ in range(N - 1):
        q = e * np.fft.ifftn(np.exp(-b * b * k2 / 6.0) * np.fft.fftn(q))
    return q


@pytest.mark.parametrize("m", CHAINS, ids=lambda m: "%dx%dx%d" % m)
def test_chain(m):
    import torch
    from ftspolysol_b200 import Engine
    from ftspolysol_b200.engine import propagate_chain_noalloc
    case = Case(name="chain", m=m, dL=0.5, species=[homopolymer("P", 4, 4, charge=0.0)], lB=0.0, ions_enabled=False)
    rng = np.random.default_rng(8)
    w = (0.3 * rng.standard_normal(m) + 0.2j * rng.standard_normal(m)).astype(np.complex128)
    wd = torch.from_numpy(w.reshape(-1)).cuda()
    q = torch.zeros_like(wd)
    eng = Engine(derive(case))
    Q = eng.propagate_chain(wd.data_ptr(), 4, 1.1, q.data_ptr())
    eng.close()
    ref = reference_chain(w, case.L, 4, 1.1)
    big = np.max(np.abs(ref))
    assert np.max(np.abs(q.cpu().numpy().reshape(m) - ref)) / big < 1e-12
    assert abs(Q - ref.mean()) / abs(ref.mean()) < 1e-12
    if max(m) <= 256 and np.prod(m) <= 262144:
        q2 = torch.full_like(wd, complex("nan"))
        rc, Q2 = propagate_chain_noalloc(m, case.L, wd.data_ptr(), 4, 1.1, q2.data_ptr())
        assert rc == 0
        assert np.max(np.abs(q2.cpu().numpy().reshape(m) - ref)) / big < 1e-12
        assert abs(Q2 - ref.mean()) / abs(ref.mean()) < 1e-12


def diblock(m):
    V = 0.125 * m[0] * m[1] * m[2]
    n = 2 * max(1, int(round(0.25 * V / 5)))
    return Case(name="ab", m=m, dL=0.5, monomer_names=["A", "B"], chi=[0.0, 0.05, 0.05, 0.0], xi=0.1, lB=1.0,
                species=[Species("AB", n, ["A", "A", "B", "B", "B"], [-1.0, -1.0, 0.0, 0.0, 1.0], [1.0, 0.9, 1.1, 1.0])],
                counterions={"number": "auto_neutralize", "valence": 1.0},
                salt={"num_salt": max(1, int(round(0.05 * V))), "cation_valence": 1.0, "anion_valence": -1.0},
                dt=0.01, stress=("xx", "yy", "zz", "xy", "xz", "yz"), isotropic_pressure=True, init_seed=6)


@pytest.mark.parametrize("m", [(9, 10, 15), (16, 25, 27), (20, 125, 6), (192, 5, 8), (48, 48, 48), (32, 32, 32)],
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
    eng = Engine(d, precision=FP64 if prec == "fp64" else FP32)
    eng.set_fields(om, ps)
    got = eng.measure(0)
    assert np.max(np.abs(eng.get("rho_type") - rho)) / np.max(np.abs(rho)) < ftol
    assert np.max(np.abs(got - rec) / np.maximum(np.abs(rec), 1e-3)) < rtol
    eng.close()
