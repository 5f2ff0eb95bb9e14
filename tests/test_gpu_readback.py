"""What ftsp_get_field may not touch: the caller's buffer before the upload
from it has finished, the step's launch count, and the state of a step in
flight."""
import ctypes as C

import numpy as np
import pytest

from ftspolysol_b200.cases import Case, homopolymer
from ftspolysol_b200.derive import derive

pytestmark = pytest.mark.gpu


def solution(m, N=4):
    V = 0.125 * m[0] * m[1] * m[2]
    return Case(name="pe", m=m, dL=0.5, monomer_names=["A"], chi=[0.0], xi=0.1, lB=1.0,
                species=[homopolymer("P", 2 * max(1, int(round(0.25 * V / N))), N)],
                counterions={"number": "auto_neutralize", "valence": 1.0}, dt=0.01, init_seed=4)


@pytest.mark.parametrize("prec", ["fp64", "fp32"])
def test_read_into_the_uploaded_buffer(prec):
    """set_fields_async(buffer), then the fields read back into that buffer:
    the upload (28 MB here) is still in flight when the read is called."""
    import torch
    from ftspolysol_b200 import Engine, FP32, FP64
    from ftspolysol_b200.engine import lib
    case = solution((96, 96, 96))
    om, ps = case.initial_fields()
    n = case.size
    host = torch.empty(4 * n, dtype=torch.float64, pin_memory=True)
    p = FP64 if prec == "fp64" else FP32
    with Engine(derive(case), precision=p) as e:
        e.set_fields(om, ps)
        ref = {k: e.get(k)[0] for k in ("omega", "psi")}
    with Engine(derive(case), precision=p) as e:
        for _ in range(4):
            host.numpy()[:] = np.concatenate([om.reshape(-1), ps.reshape(-1)]).view(np.float64)
            at = {"omega": host.data_ptr(), "psi": host.data_ptr() + 16 * n}
            e.set_fields_async_ptr(at["omega"], at["psi"])
            for k in ("psi", "omega"):
                count = C.c_longlong(0)
                assert lib().ftsp_get_field(e.h, k.encode(), C.c_void_p(at[k]), C.byref(count)) == 0
                assert count.value == 2 * n
            got = host.numpy().view(np.complex128).reshape(2, n)
            np.testing.assert_array_equal(got[0], ref["omega"])
            np.testing.assert_array_equal(got[1], ref["psi"])


@pytest.mark.parametrize("prec", ["fp64", "fp32"])
def test_reads_are_not_launches_of_the_step(prec):
    from ftspolysol_b200 import Engine, FP32, FP64
    case = solution((16, 15, 12))
    om, ps = case.initial_fields()
    with Engine(derive(case), precision=FP64 if prec == "fp64" else FP32) as e:
        e.set_fields(om, ps)
        e.step()
        n = e.launches()
        for name in ("omega", "rho_type", "psi_s"):
            e.get(name)
        assert e.launches() == n


def test_a_read_leaves_a_step_in_flight_alone():
    """A read while the batch steps returns fields of no one time, but the
    steps go on as without it."""
    from ftspolysol_b200 import Engine, FP32, SCHEME_SI
    from ftspolysol_b200.engine import Batch
    case = solution((64, 64, 64), 20)
    om, ps = case.initial_fields()
    out = []
    for read in (False, True):
        e = Engine(derive(case), precision=FP32, scheme=SCHEME_SI, noise=True, seed=3)
        e.set_fields(om, ps)
        b = Batch([e], 2)
        b.step(20)
        if read:
            for _ in range(4):
                e.get("rho_type")
        b.sync()
        out.append((e.get("omega"), e.get("psi")))
        b.close()
        e.close()
    for a, b in zip(*out):
        np.testing.assert_array_equal(a, b)
