"""Attenuation with other numbers of SLS than three: five, for which the kernels are built too, and one,
two and eight, which take the count at run time; full and at four points, with and without slices.

Compared is the stiffness of the displacement after four steps, whose stress has the memory variables
of those steps in it, against the FP64 oracle. Tolerances: a force is a sum of about 1e2 products, each
operand rounded once, so its relative 2-norm error is a few units of the working precision: 2e-6 in
float (memory variables and displacement of four steps included), 1e-13 in double. Without its memory
variables the force is off by more than 3e-5.
"""
import numpy as np
import pytest

from axisem3d_b200 import meshgen
from axisem3d_b200.solver import Solver

pytestmark = pytest.mark.gpu

TOL = {"fp32": 2e-6, "mixed": 2e-6, "fp64": 1e-13}


def _model(nsls, attenuation, is3d):
    if attenuation == "cg4":
        nrs = [30] if is3d else [11]        # the model takes one order
    else:
        nrs = [4, 17, 25, 30, 48] if is3d else [1, 8, 9, 11, 23]
    return meshgen.microbench_model(n_elem=12, nr_choices=nrs, is3d=is3d, attenuation=attenuation, nsls=nsls, seed=3)


@pytest.mark.parametrize("precision", ["fp32", "mixed", "fp64"])
@pytest.mark.parametrize("is3d", [False, True])
@pytest.mark.parametrize("attenuation", ["full", "cg4"])
@pytest.mark.parametrize("nsls", [1, 2, 5, 8])
def test_sls_counts_match_oracle(built, nsls, attenuation, is3d, precision):
    import oracle as O
    m = _model(nsls, attenuation, is3d)
    assert m.nsls == nsls
    u = meshgen.random_displacement(m, seed=4)
    o = O.Oracle(m, "fp64", threads=4)
    o.set_field(u, "displ")
    o.run(4)
    d = o.get_field("displ")
    o.compute_stiffness()
    f = o.get_field("stiff")
    rest = O.Oracle(m, "fp64", threads=4)
    rest.set_field(d, "displ")
    rest.compute_stiffness()
    assert np.linalg.norm(rest.get_field("stiff") - f) > 3e-5 * np.linalg.norm(f)
    with Solver(m, precision) as s:
        s.set_field(u, "displ")
        s.run(4)
        got = s.get_field("displ")
        s.compute_stiffness()
        g = s.get_field("stiff")
    assert np.linalg.norm(got - d) <= TOL[precision] * np.linalg.norm(d)
    assert np.linalg.norm(g - f) <= TOL[precision] * np.linalg.norm(f)
