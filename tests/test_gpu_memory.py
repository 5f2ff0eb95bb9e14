"""Device memory of a handle, counted in fields."""
import pytest

from ftspolysol_b200.cases import Case, homopolymer
from ftspolysol_b200.derive import derive

pytestmark = pytest.mark.gpu


def fields_of(d, **kw):
    import torch
    from ftspolysol_b200 import Engine
    with Engine(d, **kw):
        pass                       # context, code
    a = torch.cuda.mem_get_info()[0]
    with Engine(d, **kw):
        b = torch.cuda.mem_get_info()[0]
    return (a - b) / (16.0 * d["m"][0] * d["m"][1] * d["m"][2])


def test_scratch_of_the_transforms_is_shared():
    """A handle without electrostatics (its evaluation runs the plain
    transforms): 4 (omega) + 4 (psi) + 1 (noise) + 2 + 2 + 2 + 4 (k space) + 2
    + 1 (densities) + 1 (class table) + 4 (propagators) + 4 (scratch, the
    sweeps' two fields among them) = 31, and less than two for everything that
    does not grow with the field.  A field is 16 MiB here, a whole number of
    allocation granules."""
    m = (128, 128, 64)
    case = Case(name="chain", m=m, dL=0.5, monomer_names=["A"], chi=[0.0], xi=0.1, lB=0.0,
                species=[homopolymer("P", 4, 4, charge=0.0)], ions_enabled=False)
    assert 31.0 <= fields_of(derive(case)) < 33.0
