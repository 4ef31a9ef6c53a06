"""What handles of one process share or keep between calls: the runtime's record of an error."""
import numpy as np
import pytest

from axisem3d_b200 import meshgen
from axisem3d_b200.solver import EngineError, Solver

pytestmark = pytest.mark.gpu


def test_a_failed_call_does_not_fail_the_next_one(built):
    """The legacy default stream (address 1) cannot be captured: a run on it is refused by the host
    side of the runtime. That error is reported once, not again by the next launch of this handle or
    of another one."""
    m = meshgen.cartesian_model(nx=7, nz=5, nr=5)
    with Solver(m, "fp64") as a, Solver(m, "fp64") as b:
        b.run(4)
        a.set_stream(1)
        with pytest.raises(EngineError, match="BeginCapture"):
            a.run(4)
        b.run(4)
        a.set_stream(None)
        a.run(8)
        d, e = a.get_field("displ"), b.get_field("displ")
    # the atomic sums of 8 steps in another order
    assert np.linalg.norm(d - e) <= 1e-13 * np.linalg.norm(e)
