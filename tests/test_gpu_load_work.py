"""gmgs_load_work is the work of the loads that the last solve used."""
import numpy as np
import pytest

from gmgs import GMGSError, Solver, synthetic

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_loads_set_after_the_solve(precision):
    vox = synthetic.sphere_voids(12, 10, 16, 0, 1)
    fixed, loads = synthetic.boundary_conditions(vox, 2)
    s = Solver(vox, omega=0.4, num_levels=2, precision=precision)
    s.set_bc(fixed, loads)
    with pytest.raises(GMGSError):
        s.load_work()                                  # not solved yet
    u = s.solve()
    work = s.load_work()
    assert abs(work - s.load_vector() @ u) <= 1e-12 * abs(work)
    other = loads.copy()
    other[:, 1:] = 3 * loads[:, 1:] + 0.01
    s.set_bc(fixed, other)
    with pytest.raises(GMGSError):
        s.load_work()                                  # new loads, the displacement of the old ones
    s.stress()                                         # what needs the displacement alone still has it
    u = s.solve()
    assert abs(s.load_work() - s.load_vector() @ u) <= 1e-12 * abs(s.load_vector() @ u)
    work = s.load_work()
    with pytest.raises(GMGSError):
        s.set_bc(fixed, np.array([[10 ** 8, 0.0, 0.0, 1.0]]))     # refused: loads and solution are as before
    assert s.load_work() == work
