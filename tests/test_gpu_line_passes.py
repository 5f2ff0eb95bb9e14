"""The run-time passes: grids that have no split plan (an extent without two
radices), so that nothing else takes them.  With 243 points along x or z and a
small plane the segment pass is the plane pass; a plane of 162 x 243 points
does not fit a block, and the pass becomes y-lines, z-lines and y-lines, the
semi-implicit update runs unfused and the plain transforms take three passes.

Chain propagation against numpy FFTs (complex128, 1e-12 of the largest
modulus), densities, record and one step of either scheme of an asymmetric
chain against the oracle and the numpy restatement (complex128 1e-10;
complex64 1e-5 on fields, 2e-3 on records), the tuned launch geometry against
the default one (complex128, 1e-11): the tolerances of the split passes' tests.
"""
import functools

import numpy as np
import pytest

import pyoracle as po
from ftspolysol_b200.cases import Case, homopolymer
from ftspolysol_b200.derive import derive
from si_oracle import si_step, si_tables
from test_gpu_sizes import rec_err, rel
from test_gpu_split import diblock, reference_chain

pytestmark = pytest.mark.gpu

GRIDS = [(243, 4, 6), (4, 6, 243), (4, 162, 243)]
by_grid = pytest.mark.parametrize("m", GRIDS, ids=lambda m: "%dx%dx%d" % m)
TOL = {"fp64": (1e-10, 1e-10), "fp32": (1e-5, 2e-3)}


def precision(prec):
    from ftspolysol_b200 import FP32, FP64
    return FP64 if prec == "fp64" else FP32


@by_grid
def test_chain(m):
    import torch
    from ftspolysol_b200 import Engine
    from ftspolysol_b200.engine import propagate_chain_noalloc
    case = Case(name="chain", m=m, dL=0.5, species=[homopolymer("P", 4, 4, charge=0.0)], lB=0.0, ions_enabled=False)
    rng = np.random.default_rng(10)
    w = (0.3 * rng.standard_normal(m) + 0.2j * rng.standard_normal(m)).astype(np.complex128)
    wd = torch.from_numpy(w.reshape(-1)).cuda()
    q = torch.zeros_like(wd)
    ref = reference_chain(w, case.L, 5, 1.1)
    big = np.max(np.abs(ref))
    with Engine(derive(case)) as eng:
        Q = eng.propagate_chain(wd.data_ptr(), 5, 1.1, q.data_ptr())
    assert np.max(np.abs(q.cpu().numpy().reshape(m) - ref)) / big < 1e-12
    assert abs(Q - ref.mean()) / abs(ref.mean()) < 1e-12
    q2 = torch.full_like(wd, complex("nan"))
    rc, Q2 = propagate_chain_noalloc(m, case.L, wd.data_ptr(), 5, 1.1, q2.data_ptr())
    assert rc == 0
    assert np.max(np.abs(q2.cpu().numpy().reshape(m) - ref)) / big < 1e-12
    assert abs(Q2 - ref.mean()) / abs(ref.mean()) < 1e-12


@functools.lru_cache(maxsize=None)
def system(m):
    case = diblock(m)
    d = derive(case)
    om, ps = case.initial_fields()
    eta = np.random.default_rng(12).standard_normal((len(d["modes"]) + 1, case.size)) * 0.1
    o = po.Oracle(d)
    o.set_fields(om, ps)
    Q = o.compute_densities(0)
    rho = o.get("rho_type")
    rec = o.measure(0, Q)
    o.set_fields(om, ps)
    step = o.step(eta)[:2] + (o.get("omega"), o.get("psi"))
    o.close()
    return d, om, ps, eta, Q, rho, rec, step


@pytest.mark.parametrize("prec", ["fp64", "fp32"])
@by_grid
def test_evaluation_and_step(m, prec):
    from ftspolysol_b200 import Engine
    d, om, ps, eta, Q, rho, rec, step = system(m)
    ftol, rtol = TOL[prec]
    with Engine(d, precision=precision(prec)) as eng:
        eng.set_fields(om, ps)
        assert rel(eng.compute_densities(0), Q) < ftol
        assert rel(eng.get("rho_type"), rho) < ftol
        assert rec_err(eng.measure(0), rec) < rtol
        eng.set_fields(om, ps)
        got = eng.step(eta)
        assert rel(got[0], step[0]) < ftol
        assert rec_err(got[1], step[1]) < rtol
        assert rel(eng.get("omega"), step[2]) < ftol
        assert rel(eng.get("psi"), step[3]) < ftol


@pytest.mark.parametrize("prec", ["fp64", "fp32"])
@by_grid
def test_semi_implicit_step(m, prec):
    from ftspolysol_b200 import Engine, SCHEME_SI
    d, om, ps, eta = system(m)[:4]
    nm = len(d["modes"])
    with Engine(d, precision=precision(prec), scheme=SCHEME_SI) as eng:
        eng.set_fields(om, ps)
        om0, ps0 = eng.get("omega").reshape(nm, *m), eng.get("psi")[0].reshape(m)
        eng.step(eta)
        f = {k: eng.get(k).reshape(-1, *m) for k in ("drift", "drift_bar", "dpsi", "dpsi_bar")}
        ref = si_step(d, si_tables(d), om0, ps0, f["drift"], f["drift_bar"], f["dpsi"][0], f["dpsi_bar"][0], eta)
        for name, r in zip(("omega_bar", "psi_bar", "omega", "psi"), ref):
            assert rel(eng.get(name).reshape(r.shape), r) < TOL[prec][0], name


@by_grid
def test_tuned_geometry(m):
    from ftspolysol_b200 import Engine
    d, om, ps, eta = system(m)[:4]
    out = []
    for tune in (False, True, True):
        with Engine(d, autotune=tune) as eng:
            eng.set_fields(om, ps)
            eng.step(eta)
            out.append((eng.tune_info(), eng.get("omega"), eng.get("rho_type")))
    t0, t1, t2 = (r[0] for r in out)
    assert t0["tuned"] == 0 and t1["candidates"] >= 1 and t1["compile_time"] == 0
    assert t2["cached"] == 1 and (t2["max_radix"], t2["tile_width"]) == (t1["max_radix"], t1["tile_width"])
    for r in out[1:]:
        for a, b in zip(r[1:], out[0][1:]):
            assert np.max(np.abs(a - b)) <= 1e-11 * np.max(np.abs(b))
