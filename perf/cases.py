"""What a user of this package has it do, as timed cases.

Four kinds of call, all through the package's public entry points:

  chain    one chain propagation in a given field (Engine.propagate_chain, or
           propagate_chain_noalloc for callers that own the device memory)
  measure  the densities and the full observable record at given fields
           (Engine.measure), as an analysis of stored configurations does
  run      a block of complex-Langevin steps from given fields, the record
           read after every step (the program's own loop)
  batch    a set of independent replicas stepped as one graph

Grids have 2/3/5-smooth extents; the box has 0.5 b per grid cell.  Systems
are the package's polyelectrolyte solutions (one charged homopolymer with
counterions and salt) and block copolymers of two monomer types.
"""
import math

import numpy as np
import torch

from ftspolysol_b200 import FP32, FP64, SCHEME_PC, SCHEME_SI, Engine
from ftspolysol_b200.cases import STRESS_COMPONENTS, Case, Species, polyelectrolyte_case
from ftspolysol_b200.derive import derive
from ftspolysol_b200.engine import Batch, propagate_chain_noalloc
from ftspolysol_b200.replicas import CHAIN_LENGTHS, GRIDS

SMOOTH = sorted(2**a * 3**b * 5**c for a in range(8) for b in range(5) for c in range(4) if 8 <= 2**a * 3**b * 5**c <= 128)


def _chain(m1, m2, m3, N, b, noalloc=False):
    return {"kind": "chain", "m1": m1, "m2": m2, "m3": m3, "N": N, "b": b, "noalloc": noalloc}


def _system(kind, prec, m1, m2, m3, N, chain, **more):
    d = {"kind": kind, "prec": prec, "m1": m1, "m2": m2, "m3": m3, "N": N, "chain": chain, "valence": 1.0, "salt": 0.1,
         "stress": True}
    d.update(more)
    return d


def _run(prec, scheme, m1, m2, m3, N, steps, chain="homo", noise=True, mode="plain", **more):
    return _system("run", prec, m1, m2, m3, N, chain, scheme=scheme, steps=steps, noise=noise, mode=mode, **more)


def listed():
    return [
        # a framework's inner loop calling the allocation-free propagation on a small ragged mesh
        dict(_chain(24, 20, 18, 12, 1.0, noalloc=True), name="chain_noalloc_24x20x18"),
        # a mesh of mixed factors, larger than one block's memory in a plane
        dict(_chain(90, 125, 100, 40, 1.2), name="chain_90x125x100"),
        # the production mesh in complex128
        dict(_chain(128, 128, 128, 50, 1.0), name="chain_128"),
        # analysis of a stored configuration: diblock copolymer, both sweeps, complex64
        dict(_system("measure", "fp32", 64, 64, 64, 50, "diblock"), name="measure_64_diblock_fp32"),
        # the same of a homopolymer solution on a ragged mesh, complex128
        dict(_system("measure", "fp64", 60, 48, 40, 32, "homo"), name="measure_60x48x40_fp64"),
        # validation runs: the smallest production box, complex128, the reference's scheme
        dict(_run("fp64", "pc", 32, 32, 32, 32, 40), name="run_32_fp64_pc"),
        # production runs at 64^3 with the guards that long runs use (adaptive step, device checkpoints)
        dict(_run("fp32", "si", 64, 64, 64, 50, 20, mode="guarded"), name="run_64_fp32_si"),
        # a medium box on a mixed-radix mesh with the learned preconditioner collecting and in use
        dict(_run("fp32", "si", 48, 48, 48, 32, 10, mode="learned"), name="run_48_fp32_learned"),
        # a mixed-radix box of the replica sweep
        dict(_run("fp32", "si", 96, 96, 96, 32, 10), name="run_96_fp32_si"),
        # the headline system: 128^3, N = 50, divalent counterions, full stress
        dict(_run("fp32", "si", 128, 128, 128, 50, 10, valence=2.0, salt=0.05), name="run_128_fp32_si"),
        # the same in complex128 with the reference's scheme, without noise (relaxation to a saddle point)
        dict(_run("fp64", "pc", 128, 128, 128, 50, 3, valence=2.0, salt=0.05, noise=False), name="run_128_fp64_pc"),
        # a replica sweep: uneven grids, chain lengths and salt, one graph
        {"kind": "batch", "name": "batch_16", "replicas": 16, "steps": 4, "system_seed": 2024},
    ]


def draw(rng):
    def extent(lo, hi):
        want = math.exp(rng.uniform(math.log(lo), math.log(hi)))
        return min((n for n in SMOOTH if lo <= n <= hi), key=lambda n: abs(math.log(n / want)))

    kind = rng.choice(["chain", "chain", "measure", "run", "run", "run", "batch"])
    if kind == "chain":
        if rng.random() < 0.3:
            return _chain(extent(8, 64), extent(8, 64), extent(8, 64), int(math.exp(rng.uniform(math.log(2), math.log(50)))),
                          round(rng.uniform(0.8, 1.4), 3), noalloc=True)
        return _chain(extent(16, 128), extent(16, 128), extent(16, 128), int(math.exp(rng.uniform(math.log(4), math.log(50)))),
                      round(rng.uniform(0.8, 1.4), 3))
    if kind == "batch":
        return {"kind": "batch", "replicas": 4 * rng.randint(1, 4), "steps": rng.randint(1, 4), "system_seed": rng.randint(1, 10**6)}
    prec = rng.choice(["fp32", "fp32", "fp64"])
    chain = rng.choice(["homo", "homo", "homo", "diblock", "triblock"])
    scheme = rng.choice(["si", "si", "pc"])
    mode = rng.choice(["plain", "plain", "guarded", "learned"]) if kind == "run" and scheme == "si" else "plain"
    largest = 64 if mode == "learned" else 128
    if rng.random() < 0.5:
        m1 = m2 = m3 = extent(16, largest)
    else:
        m1, m2, m3 = extent(16, largest), extent(16, largest), extent(16, largest)
    N = int(math.exp(rng.uniform(math.log(6), math.log(50))))
    more = {"valence": rng.choice([1.0, 2.0]), "salt": round(rng.uniform(0.01, 0.3), 3), "stress": rng.random() < 0.7}
    if kind == "measure":
        return _system("measure", prec, m1, m2, m3, N, chain, **more)
    noise = rng.random() < 0.8
    cost = m1 * m2 * m3 * N * (2 if chain == "diblock" else 1) * (2 if prec == "fp64" else 1)
    steps = min(rng.randint(1, 10), max(1, 96**3 * 320 // cost))   # no more work than the listed ones
    return _run(prec, scheme, m1, m2, m3, N, steps, chain=chain, noise=noise, mode=mode, **more)


# ---- systems ----
def _model(case):
    """The derived numbers of a case's system (what a param file states)."""
    m = (case["m1"], case["m2"], case["m3"])
    N = case["N"]
    V = 0.125 * m[0] * m[1] * m[2]
    z = int(case["valence"])
    stress = STRESS_COMPONENTS if case["stress"] else ()
    chains = z * max(1, round(0.5 * V / N / z))   # divisible: the counterions neutralise exactly
    salt = {"num_salt": round(case["salt"] * V), "cation_valence": 1.0, "anion_valence": -1.0}
    ions = {"counterions": {"number": "auto_neutralize", "valence": case["valence"]}, "salt": salt if salt["num_salt"] else None}
    half = max(1, N // 2)
    third = max(1, N // 3)
    if case["chain"] == "homo":
        mono, charge, types, chi = ["A"] * N, [-1.0] * N, ["A"], [0.0]
    elif case["chain"] == "diblock":   # a charged and a neutral block
        mono, charge = ["A"] * half + ["B"] * (N - half), [-1.0] * half + [0.0] * (N - half)
        types, chi = ["A", "B"], [0.0, 0.04, 0.04, 0.0]
    else:   # mirror-symmetric: charged ends, neutral middle
        mono, charge = ["A"] * third + ["B"] * (N - 2 * third) + ["A"] * third, [-1.0] * third + [0.0] * (N - 2 * third) + [-1.0] * third
        types, chi = ["A", "B"], [0.0, 0.04, 0.04, 0.0]
    return derive(Case(name="perf", m=m, dL=0.5, a=1.0, monomer_names=types, chi=chi, xi=0.1, lB=1.0,
                       species=[Species("P", chains, mono, charge)], dt=0.005, stress=stress,
                       isotropic_pressure=bool(stress), **ions))


def _fields(n_modes, size, seed):
    """Fields a run starts from: white noise of the package's usual size,
    with small imaginary parts."""
    rng = np.random.default_rng(seed)
    om = torch.empty((n_modes, size), dtype=torch.complex128, pin_memory=True)
    ps = torch.empty(size, dtype=torch.complex128, pin_memory=True)
    for f in [om[a] for a in range(n_modes)] + [ps]:
        f.copy_(torch.complex(torch.from_numpy(0.1 * rng.standard_normal(size)), torch.from_numpy(0.01 * rng.standard_normal(size))))
    return om, ps


class _View:
    """A device array of the engine as torch sees it (torch keeps this
    object, and so the engine, for as long as the tensor lives)."""

    def __init__(self, engine, ptr, shape):
        self.engine = engine
        self.__cuda_array_interface__ = {"data": (int(ptr), False), "shape": shape, "typestr": "<c16", "version": 3}


def _prec(case):
    return FP32 if case["prec"] == "fp32" else FP64


def _typed(case, a):
    """Results in the type the engine computes them in."""
    a = np.asarray(a)
    if case["prec"] == "fp64":
        return a
    return a.astype(np.complex64 if a.dtype.kind == "c" else np.float32)


def _chain_inputs(case, seed):
    n = case["m1"] * case["m2"] * case["m3"]
    g = torch.Generator("cuda").manual_seed(seed)
    w = torch.complex(0.3 * torch.randn(n, dtype=torch.float64, device="cuda", generator=g),
                      0.2 * torch.randn(n, dtype=torch.float64, device="cuda", generator=g))
    return w


def prepare(case, seed):
    s = {"case": case}
    if case["kind"] == "chain":
        s["w"] = _chain_inputs(case, seed)
        s["q"] = torch.zeros_like(s["w"])
        s["m"] = (case["m1"], case["m2"], case["m3"])
        s["L"] = tuple(0.5 * v for v in s["m"])
        if not case["noalloc"]:
            s["eng"] = Engine(derive(Case(name="chain", m=s["m"], dL=0.5, species=[Species("P", 4, ["A"] * 4, [0.0] * 4)],
                                          lB=0.0, ions_enabled=False)))
        return s
    if case["kind"] == "batch":
        rng = np.random.default_rng(case["system_seed"])
        s["engines"], s["fields"] = [], []
        R = case["replicas"]
        for r in range(R):
            m = GRIDS[r * len(GRIDS) // R]
            d = derive(polyelectrolyte_case("rep", m, int(rng.choice(CHAIN_LENGTHS)), 1.0, float(rng.uniform(0.01, 0.5)),
                                            isotropic_pressure=True))
            s["engines"].append(Engine(d, precision=FP32, scheme=SCHEME_SI, noise=True, seed=seed * 1000 + r))
            s["fields"].append(_fields(1, m**3, seed * 1000 + r))
        for e, (om, ps) in zip(s["engines"], s["fields"]):
            e.set_fields_ptr(om.data_ptr(), ps.data_ptr())
        s["batch"] = Batch(s["engines"])
        return s
    d = _model(case)
    size = case["m1"] * case["m2"] * case["m3"]
    s["om"], s["ps"] = _fields(len(d["modes"]), size, seed)
    if case["kind"] == "measure":
        s["eng"] = Engine(d, precision=_prec(case))
        return s
    guard = {"restart_interval": 100} if case["mode"] == "guarded" else {}
    e = s["eng"] = Engine(d, precision=_prec(case), scheme=SCHEME_SI if case["scheme"] == "si" else SCHEME_PC,
                          noise=case["noise"], seed=seed, **guard)
    if case["mode"] == "guarded":
        e.set_adaptive(300.0)
    if case["mode"] == "learned":   # weights as a file would give them
        e.learn_configure(N=case["N"], lB=1.0, salt=case["salt"], seed=7)
        rng = np.random.default_rng(seed)
        e.learn_set_weights((0.05 * rng.standard_normal(e.learn_weights().size)).astype(np.float32))
        e.learn_collect(True)
        e.learn_use(True)
    if case["prec"] == "fp64":
        v = e.views()
        shape = (len(d["modes"]), size)
        s["state"] = [torch.as_tensor(_View(e, v.omega, shape), device="cuda"), torch.as_tensor(_View(e, v.psi, (size,)), device="cuda")]
    return s


def run(s):
    case = s["case"]
    if case["kind"] == "chain":
        if case["noalloc"]:
            rc, Q = propagate_chain_noalloc(s["m"], s["L"], s["w"].data_ptr(), case["N"], case["b"], s["q"].data_ptr())
            if rc:
                raise RuntimeError("propagate_chain_noalloc: status %d" % rc)
        else:
            Q = s["eng"].propagate_chain(s["w"].data_ptr(), case["N"], case["b"], s["q"].data_ptr())
        return {"Q": np.array(Q), "q": s["q"]}
    if case["kind"] == "batch":
        for e, (om, ps) in zip(s["engines"], s["fields"]):
            e.set_fields_ptr(om.data_ptr(), ps.data_ptr())
        s["batch"].step(case["steps"])
        s["batch"].sync()
        out = {}
        for r, e in enumerate(s["engines"]):
            _, rec, dmax = e.read_status()
            out["%02d" % r] = np.concatenate([rec.real, rec.imag, dmax]).astype(np.float32)
        return out
    e = s["eng"]
    e.set_fields_async_ptr(s["om"].data_ptr(), s["ps"].data_ptr())
    if case["kind"] == "measure":
        rec = e.measure(0)
        return {"record": _typed(case, rec), "rho": _typed(case, e.get("rho_type"))}
    Qs, recs, dmaxs = zip(*(e.step() for _ in range(case["steps"])))
    if case["prec"] == "fp64":
        om, ps = s["state"]
    else:   # the checkpoint fields
        om, ps = _typed(case, e.get("omega")), _typed(case, e.get("psi"))
    return {"Q": _typed(case, Qs), "record": _typed(case, recs), "drift_max": _typed(case, dmaxs), "omega": om, "psi": ps}


def work(case):
    """One segment step reads a propagator and the segment factor and writes
    the next propagator and is a forward and an inverse 3-D transform; a
    mirror-symmetric chain needs one sweep, others two; the fields of a step
    are read and written a few times more."""
    if case["kind"] == "batch":
        rng = np.random.default_rng(case["system_seed"])
        b = f = 0.0
        for r in range(case["replicas"]):
            m = GRIDS[r * len(GRIDS) // case["replicas"]]
            N = int(rng.choice(CHAIN_LENGTHS))
            rng.uniform(0.01, 0.5)
            b += case["steps"] * 2 * (N + 10) * 8 * m**3
            f += case["steps"] * 2 * N * 10 * m**3 * math.log2(m**3)
        return {"bytes": b, "flops": f}
    V = case["m1"] * case["m2"] * case["m3"]
    sc = 16 if case["kind"] == "chain" or case["prec"] == "fp64" else 8
    flops = 10.0 * V * math.log2(V)   # a forward and an inverse transform
    if case["kind"] == "chain":
        return {"bytes": 2.0 * sc * V, "flops": (case["N"] - 1) * flops}
    sweeps = 2 if case["chain"] == "diblock" else 1
    evals = 1 if case["kind"] == "measure" else 2 * case["steps"]
    # stored propagators written and read once each, plus the fields around them
    return {"bytes": evals * (2.0 * case["N"] + 10) * sc * V, "flops": evals * (sweeps * case["N"] + 5) * flops}


# ---- the same in 64 bits with torch ----
def _waves(m, L):
    ks = []
    for n, l in zip(m, L):
        i = torch.arange(n, dtype=torch.float64, device="cuda")
        ks.append(2 * math.pi * torch.where(i > n // 2, i - n, i) / l)
    return ks[0][:, None, None], ks[1][None, :, None], ks[2][None, None, :]


def _conv(x, f):
    return torch.fft.ifftn(torch.fft.fftn(x) * f)


class _Exact:
    """Densities, drifts, observables and steps of one system."""

    def __init__(self, d):
        self.d, self.m = d, tuple(d["m"])
        self.k = _waves(self.m, d["L"])
        self.k2 = sum(k * k for k in self.k)
        self.V = float(np.prod(d["L"]))
        self.n = int(np.prod(self.m))
        self.gam = torch.exp(-0.5 * d["a"] ** 2 * self.k2)

    def flip(self, x):   # x(-k)
        return torch.roll(torch.flip(x, (0, 1, 2)), (1, 1, 1), (0, 1, 2))

    def eval(self, om, ps, observe):
        d, gam = self.d, self.gam
        pk = torch.fft.fftn(ps)
        ok = [torch.fft.fftn(w) for w in om]
        wk = [gam * sum(md["gamma"] * md["O"][t] * o for md, o in zip(d["modes"], ok)) for t in range(d["M"])]
        W = [torch.fft.ifftn(w) for w in wk]
        psi_s = torch.fft.ifftn(gam * pk)
        raw = [torch.zeros_like(ps) for _ in range(d["M"])]
        raw_c = torch.zeros_like(ps)
        kk = [(0, 0), (1, 1), (2, 2), (0, 1), (0, 2), (1, 2)]
        kprod = [self.k[a] * self.k[b] for a, b in kk]
        conn = [0.0] * 6
        self.Q = []
        for sp in d["species"]:
            N = len(sp["types"])
            E = [None] * N
            made = {}
            for s in range(N):
                key = (sp["types"][s], sp["charges"][s])
                if key not in made:
                    made[key] = torch.exp(-(W[key[0]] + 1j * key[1] * psi_s))
                E[s] = made[key]
            phi = {b: torch.exp(-b * b * self.k2 / 6.0) for b in set(sp["bonds"])}
            q = [E[0]]
            for s in range(N - 1):
                q.append(E[s + 1] * _conv(q[s], phi[sp["bonds"][s]]))
            Q = q[-1].mean()
            self.Q.append(Q)
            fac = sp["num_chains"] / self.V / Q
            b = E[N - 1]
            for s in range(N - 1, -1, -1):
                rho = fac * q[s] * b / E[s]
                raw[sp["types"][s]] += rho
                raw_c += sp["charges"][s] * rho
                if s > 0:
                    bl = sp["bonds"][s - 1]
                    bk = torch.fft.fftn(b)
                    if observe:
                        t = bl * bl * fac * phi[bl] * torch.fft.fftn(q[s - 1]) * self.flip(bk)
                        for c in range(6):
                            conn[c] += (kprod[c] * t).sum()
                    b = E[s - 1] * torch.fft.ifftn(bk * phi[bl])
        self.rho = [_conv(r, gam) for r in raw]
        rho_c = _conv(raw_c, gam)
        self.Qion, ion_k = [], []
        for i in d["ions"]:
            gj = torch.exp(-0.5 * i["smear"] ** 2 * self.k2)
            f = torch.exp(-1j * i["valence"] * torch.fft.ifftn(gj * pk))
            Qj = f.mean()
            self.Qion.append(Qj)
            f = torch.fft.fftn(f * (i["count"] / self.V / Qj))
            rho_c = rho_c + i["valence"] * torch.fft.ifftn(gj * f)
            ion_k.append((i, gj, f))
        self.dpsi = torch.fft.ifftn(self.k2 * pk) / (4 * math.pi * d["lB"]) + 1j * rho_c
        self.u = [md["coeff"] * w + sum(md["gamma"] * md["O"][t] * self.rho[t] for t in range(d["M"])) for md, w in zip(d["modes"], om)]
        return self.observe(om, pk, wk, raw, raw_c, ion_k, kprod, conn) if observe else None

    def observe(self, om, pk, wk, raw, raw_c, ion_k, kprod, conn):
        d, n2 = self.d, float(self.n) ** 2
        sp, ions = d["species"], d["ions"]
        mu = [-torch.log(q) for q in self.Q] + [-torch.log(q) for q in self.Qion]
        count = [s["num_chains"] for s in sp] + [i["count"] for i in ions]
        rec = list(mu)
        for s in sp:
            rec.append(-d["lB"] * sum(z * z for z in s["charges"]) / (2 * math.sqrt(math.pi) * d["a"]))
        for i in ions:
            rec.append(-d["lB"] * i["valence"] ** 2 / (2 * math.sqrt(math.pi) * i["smear"]))
        rec += [math.log(c / self.V) for c in count]
        X = pk * self.flip(pk)
        Xc = [(kp * X).sum() for kp in kprod]
        Xtr = Xc[0] + Xc[1] + Xc[2]
        H = sum(0.5 * md["coeff"] * (w * w).mean() for md, w in zip(d["modes"], om)) + Xtr / (8 * math.pi * d["lB"] * n2)
        rec.append(H + sum(c / self.V * m for c, m in zip(count, mu)))
        if d["stress"]:
            A = sum(self.flip(torch.fft.fftn(r)) * w for r, w in zip(raw, wk))
            B = 1j * self.flip(torch.fft.fftn(raw_c)) * self.gam * pk
            base, v0 = -d["a"] ** 2 * (A + B), 0.5 * A + B / 6
            for i, gj, f in ion_k:
                ip = 1j * i["valence"] * self.flip(f) * gj * pk
                base, v0 = base - i["smear"] ** 2 * ip, v0 + ip / 6
            F = [(kp * base).sum() for kp in kprod]
            v0 = v0.sum()
            ideal = sum(count) / self.V + d["self_pressure"]
            some = self.k2 > 0
            inv = torch.where(some, 1.0 / torch.where(some, self.k2, torch.ones_like(self.k2)), torch.zeros_like(self.k2))
            for c, name in enumerate(STRESS_COMPONENTS):
                if name not in d["stress"]:
                    continue
                delta = 1.0 if c < 3 else 0.0
                v = ideal * delta + (delta * float(some.sum()) / 3.0 - float((kprod[c] * inv).sum())) / self.V
                v = v + (Xc[c] - delta * Xtr / 3) / (4 * math.pi * d["lB"] * n2) + conn[c] / (3 * n2) + (F[c] + delta * v0) / n2
                rec.append(v)
            if d["isotropic_pressure"]:
                rec.append(ideal + (conn[0] + conn[1] + conn[2]) / (9 * n2) + ((F[0] + F[1] + F[2]) / 3 + v0) / n2)
        return np.array([complex(r) for r in rec])

    def response(self):
        """Linear response of the drifts of the homogeneous state, per field."""
        d = self.d
        out = []
        for md in d["modes"]:
            out.append(torch.clamp(md["coeff"] - (complex(md["gamma"]) ** 2).real * self.gam**2 * self.corr([[md["O"][t] for t in sp["types"]] for sp in d["species"]]), min=0.0))
        G = self.k2 / (4 * math.pi * d["lB"]) + self.gam**2 * self.corr([sp["charges"] for sp in d["species"]])
        for i in d["ions"]:
            G = G + i["count"] / self.V * i["valence"] ** 2 * torch.exp(-i["smear"] ** 2 * self.k2)
        return out + [torch.where(self.k2 > 0, G, torch.zeros_like(G))]

    def corr(self, weights):
        S = torch.zeros_like(self.k2)
        for sp, w in zip(self.d["species"], weights):
            F = torch.zeros_like(self.k2)
            for s, x in enumerate(w):
                if s:
                    F = F * torch.exp(-sp["bonds"][s - 1] ** 2 * self.k2 / 6)
                S += sp["num_chains"] / self.V * x * (x + 2 * F)
                F = F + x
        return torch.where(self.k2 > 0, S, torch.zeros_like(S))

    def steps(self, om, ps, count, implicit):
        d, dt = self.d, self.d["dt"]
        lam = [md["lambda"] for md in d["modes"]] + [d["lambda_psi"]]
        P = [1.0 / (1.0 + dt * l * g) for l, g in zip(lam, self.response())] if implicit else [1.0] * len(lam)
        Qs, recs, dmaxs = [], [], []
        mean0 = lambda x: x - x.mean()  # noqa: E731
        for _ in range(count):
            self.eval(om, ps, False)
            u0 = self.u + [mean0(self.dpsi)]
            now = om + [ps]
            bar = [w + _conv(-dt * l * u, p) for w, l, u, p in zip(now, lam, u0, P)]
            bar[-1] = mean0(bar[-1])
            recs.append(self.eval(bar[:-1], bar[-1], True))
            Qs.append([complex(q) for q in self.Q])
            u1 = self.u + [mean0(self.dpsi)]
            dmaxs.append([abs(0.5 * l) * float((a + b).abs().max()) for l, a, b in zip(lam, u0, u1)])
            new = [w + _conv(-0.5 * dt * l * (a + b), p) for w, l, a, b, p in zip(now, lam, u0, u1, P)]
            om, ps = new[:-1], mean0(new[-1])
        return {"Q": np.array(Qs), "record": np.array(recs), "drift_max": np.array(dmaxs), "omega": torch.stack(om).reshape(len(om), -1),
                "psi": ps.reshape(-1)}


def exact(case, seed):
    if case["kind"] == "chain":
        m = (case["m1"], case["m2"], case["m3"])
        E = torch.exp(-_chain_inputs(case, seed)).reshape(m)
        k = _waves(m, tuple(0.5 * v for v in m))
        phi = torch.exp(-case["b"] ** 2 * sum(x * x for x in k) / 6)
        q = E
        for _ in range(case["N"] - 1):
            q = E * _conv(q, phi)
        return {"Q": np.array(complex(q.mean())), "q": q.reshape(-1)}
    # generated noise, and a network in the loop, have no plain value
    if case["kind"] == "batch" or case["kind"] == "run" and (case["noise"] or case["mode"] == "learned"):
        return None
    d = _model(case)
    om, ps = _fields(len(d["modes"]), int(np.prod(d["m"])), seed)
    om = [w.cuda().reshape(d["m"]) for w in om]
    ps = ps.cuda().reshape(d["m"])
    ps = ps - ps.mean()
    x = _Exact(d)
    if case["kind"] == "measure":
        return {"record": x.eval(om, ps, True), "rho": torch.stack(x.rho).reshape(d["M"], -1)}
    out = x.steps(om, ps, case["steps"], case["scheme"] == "si")
    if case["prec"] == "fp32":   # handed out as host arrays
        out["omega"], out["psi"] = out["omega"].cpu().numpy(), out["psi"].cpu().numpy().reshape(1, -1)
    return out
