"""A long porous column: more nodes on stored matrices than the z layers of one launch hold.

The down-sweep of a mixed level takes those nodes as grid layers before its tiles;
60 x 12 elements make one tile of 31 x 7 nodes on level 2, so each plane there needs
about 7 layers, and 9700 planes more than the 65535 a launch may have.  The
preconditioner of the FP64 handle is the reference (FP32 rounding: 1e-4 relative is
far above its error and far below that of a missing part)."""
import numpy as np
import pytest

from gmgs import Solver

pytestmark = pytest.mark.gpu


def test_preconditioner_of_a_long_column():
    ny, nx, nz = 60, 12, 19400
    vox = np.ones((ny, nx, nz), dtype=np.int32, order="F")
    vox[1::2, 1::2, 401::2] = 0                         # one voxel missing of every 2 x 2 x 2
    plane = (ny + 1) * (nx + 1)
    fixed = np.arange(1, plane + 1, dtype=np.int32)
    loads = np.array([[plane + 1, 0.0, 0.0, -1.0]])
    r = None
    out = []
    for precision in ("fp64", "mixed"):
        s = Solver(vox, omega=0.4, num_levels=3, precision=precision)
        s.set_bc(fixed, loads)
        if r is None:
            r = np.random.default_rng(2).standard_normal(3 * s.num_nodes(1))
            r[:3 * plane] = 0
        out.append(s.apply_preconditioner(r))
        s.close()
    assert np.linalg.norm(out[1] - out[0]) <= 1e-4 * np.linalg.norm(out[0])
