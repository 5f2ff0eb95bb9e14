"""Backward sweep, stress sums and field transforms of the compile-time passes
at 64, 96 and 128 cubed (an asymmetric chain, which runs both sweeps and the
plain transforms; the stress variant of the two-exchange k-space pass at 96
and 128), and one step of either scheme at 96 cubed, in both precisions.

Checked against the oracle and, for the semi-implicit step, the numpy
restatement, with the tolerances of test_gpu_sizes.py and test_gpu_si.py:
1e-10 in complex128; in complex64 1e-5 on fields and 2e-3 on records.
"""
import functools

import numpy as np
import pytest

import pyoracle as po
from ftspolysol_b200.derive import derive
from si_oracle import si_step, si_tables
from test_gpu_sizes import pe_case, rec_err, rel
from test_gpu_split import diblock

pytestmark = pytest.mark.gpu

TOL = {"fp64": (1e-10, 1e-10), "fp32": (1e-5, 2e-3)}


def precision(prec):
    from ftspolysol_b200 import FP32, FP64
    return FP64 if prec == "fp64" else FP32


@functools.lru_cache(maxsize=1)
def oracle_measure(n):
    case = diblock((n, n, n))
    d = derive(case)
    om, ps = case.initial_fields()
    o = po.Oracle(d)
    o.set_fields(om, ps)
    Q = o.compute_densities(0)
    out = d, om, ps, Q, o.get("rho_type"), o.measure(0, Q)
    o.close()
    return out


@pytest.mark.parametrize("prec", ["fp64", "fp32"])
@pytest.mark.parametrize("n", [64, 96, 128])
def test_both_sweeps(n, prec):
    from ftspolysol_b200 import Engine
    d, om, ps, Q, rho, rec = oracle_measure(n)
    ftol, rtol = TOL[prec]
    with Engine(d, precision=precision(prec)) as eng:
        eng.set_fields(om, ps)
        assert rel(eng.compute_densities(0), Q) < ftol
        assert rec_err(eng.measure(0), rec) < rtol
        assert rel(eng.get("rho_type"), rho) < ftol


@functools.lru_cache(maxsize=1)
def oracle_step():
    case = pe_case((96, 96, 96), 4)
    d = derive(case)
    om, ps = case.initial_fields()
    eta = np.random.default_rng(11).standard_normal((2, case.size)) * 0.2
    o = po.Oracle(d)
    o.set_fields(om, ps)
    Q, rec, _ = o.step(eta)
    out = d, om, ps, eta, Q, rec, o.get("omega"), o.get("psi")
    o.close()
    return out


@pytest.mark.parametrize("prec", ["fp64", "fp32"])
def test_step_96(prec):
    from ftspolysol_b200 import Engine
    d, om, ps, eta, Qo, reco, omo, pso = oracle_step()
    ftol, rtol = TOL[prec]
    with Engine(d, precision=precision(prec)) as eng:
        eng.set_fields(om, ps)
        Q, rec, _ = eng.step(eta)
        assert rel(Q, Qo) < ftol
        assert rec_err(rec, reco) < rtol
        assert rel(eng.get("omega"), omo) < ftol
        assert rel(eng.get("psi"), pso) < ftol


@pytest.mark.parametrize("prec", ["fp64", "fp32"])
def test_semi_implicit_step_96(prec):
    from ftspolysol_b200 import Engine, SCHEME_SI
    d, om, ps, eta = oracle_step()[:4]
    m = tuple(d["m"])
    ftol = TOL[prec][0]
    with Engine(d, precision=precision(prec), scheme=SCHEME_SI) as eng:
        eng.set_fields(om, ps)
        om0, ps0 = eng.get("omega").reshape(1, *m), eng.get("psi")[0].reshape(m)
        eng.step(eta)
        f = {k: eng.get(k).reshape(-1, *m) for k in ("drift", "drift_bar", "dpsi", "dpsi_bar")}
        ref = si_step(d, si_tables(d), om0, ps0, f["drift"], f["drift_bar"], f["dpsi"][0], f["dpsi_bar"][0], eta)
        for name, r in zip(("omega_bar", "psi_bar", "omega", "psi"), ref):
            assert rel(eng.get(name).reshape(r.shape), r) < ftol, name
