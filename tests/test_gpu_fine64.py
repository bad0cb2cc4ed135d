"""FP64 operator kernels (fine64.cu) at the sizes where their tiling can go
wrong, against the oracle: node counts around the 32 x 8 tile and the z-chunk
edges, voxels that are not cubes, boundary and void nodes (node lists), levels
with stored matrices, and the scaled elements of a density field.

Tolerance: a row sums fewer than 700 products; on a random vector |K||x| is of
the order of |K x|, so the relative error stays below 700 * 2^-53 = 8e-14 in
any summation order, on either side."""
import numpy as np
import pytest

from gmgs import Solver, synthetic
from gmgs_oracle import Oracle, Params

pytestmark = pytest.mark.gpu

TOL = 2e-13


def rel(a, b):
    return np.linalg.norm(a - b) / np.linalg.norm(b)


def pair(shape, voids, levels, ele, rho_range, seed):
    nely, nelx, nelz = shape
    vox = synthetic.sphere_voids(nelx, nely, nelz, voids, seed)
    fixed, loads = synthetic.boundary_conditions(vox, levels)
    o = Oracle(vox, Params(omega=0.4, num_levels=levels), ele_size=ele)
    o.apply_boundary_condition(fixed, loads)
    s = Solver(vox, ele_size=ele, omega=0.4, num_levels=levels)
    s.set_bc(fixed, loads)
    if rho_range:
        rho = synthetic.density(int(vox.sum()), rho_range, seed)
        o.set_density(rho, 3.0)
        s.set_density(rho, 3.0)
    return o, s


# (ny, nx, nz) elements: node counts one below, at and one above the tile, and beyond it
@pytest.mark.parametrize("rho_range", [None, (0.2, 1.0)], ids=["uniform", "density"])
@pytest.mark.parametrize("shape,voids,levels,ele", [
    ((4, 4, 4), 0, 2, (1.0, 1.0, 1.0)),
    ((30, 6, 10), 0, 2, (1.0, 1.0, 1.0)),
    ((32, 8, 12), 0, 2, (0.9, 1.1, 1.3)),
    ((34, 10, 14), 2, 2, (1.0, 1.0, 1.0)),
    ((20, 18, 70), 6, 3, (1.02, 0.97, 1.0)),
    ((63, 15, 33), 4, 3, (1.0, 1.0, 1.0)),
])
def test_operator_and_vcycle_match_oracle(shape, voids, levels, ele, rho_range):
    o, s = pair(shape, voids, levels, ele, rho_range, 17)
    o.setup()
    rng = np.random.default_rng(3)
    for l, lv in enumerate(o.levels):
        x = rng.standard_normal(lv.numDOFs)
        assert rel(s.apply_operator(x, l + 1), o.atx(x, l)) < TOL, f"level {l + 1}"
    r = rng.standard_normal(o.levels[0].numDOFs)
    r[o.levels[0].fixedDOFs] = 0
    assert rel(s.apply_preconditioner(r), o.vcycle(r)) < 1e-10


def test_operator_on_a_mixed_handle_matches_the_fp64_one():
    """A mixed handle builds what the FP64 operator needs when it is first applied."""
    vox = synthetic.sphere_voids(28, 21, 36, 3, 4)
    fixed, loads = synthetic.boundary_conditions(vox, 3)
    rng = np.random.default_rng(5)
    handles = []
    for precision in ("fp64", "mixed"):
        s = Solver(vox, omega=0.4, num_levels=3, precision=precision)
        s.set_bc(fixed, loads)
        s.solve()
        handles.append(s)
    for level in (1, 2, 3):
        x = rng.standard_normal(3 * handles[0].num_nodes(level))
        assert np.array_equal(handles[0].apply_operator(x, level), handles[1].apply_operator(x, level))
