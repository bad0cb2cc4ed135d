"""A launch that CUDA refuses fails its own call and no other."""
import numpy as np
import pytest

from gmgs import GMGSError, Solver, synthetic

pytestmark = pytest.mark.gpu


def test_refused_launch_then_another_handle():
    # 70001 planes on the coarse level: more than the z extent of a grid
    vox = np.ones((2, 2, 140000), dtype=np.int32, order="F")
    s = Solver(vox, omega=0.4, num_levels=2)
    s.set_bc(np.arange(1, 10), np.array([[10, 0.0, 0.0, -1.0]]))
    with pytest.raises(GMGSError, match="(?i)launch"):
        s.solve()
    s.close()
    vox = synthetic.sphere_voids(8, 8, 8, 0, 1)
    s = Solver(vox, omega=0.4, num_levels=2)
    s.set_bc(*synthetic.boundary_conditions(vox, 2))
    assert np.isfinite(s.solve()).all() and s.status == 0
