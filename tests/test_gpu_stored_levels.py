"""Mixed down-sweep of levels whose nodes all lie on stored matrices (a density
model's coarse levels): up to one wave of CTAs (32 nodes each, 5 CTAs on 152 SMs:
24320 nodes) and beyond take different orders of loads.  Level 2 here has 31 x 31
nodes on 25 and on 26 planes.  Against the FP64 handle: FP32 rounding through a
V-cycle stays below 1e-5 of the result, a missing node or element does not."""
import numpy as np
import pytest

from gmgs import Solver, synthetic

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nz", [48, 50])
def test_preconditioner_matches_fp64(nz):
    vox = synthetic.sphere_voids(60, 60, nz, 0, 1)
    fixed, loads = synthetic.boundary_conditions(vox, 2)
    rho = synthetic.density(int(vox.sum()), (0.2, 1.0), 4)
    r = np.random.default_rng(6).standard_normal(3 * 61 * 61 * (nz + 1))
    r[:3 * 61 * 61] = 0
    out = []
    for precision in ("fp64", "mixed"):
        s = Solver(vox, omega=0.4, num_levels=3, precision=precision)
        s.set_bc(fixed, loads)
        s.set_density(rho, 3.0)
        assert s.num_nodes(2) == 31 * 31 * (nz // 2 + 1)
        out.append(s.apply_preconditioner(r))
    assert np.linalg.norm(out[1] - out[0]) <= 1e-5 * np.linalg.norm(out[0])
