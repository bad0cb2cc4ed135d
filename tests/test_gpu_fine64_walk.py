"""The z walk of the FP64 kernels: chunks of more than one plane.

A CTA walks a chunk of planes whose length follows from the size of the grid, so
a part in the corner of a larger, empty box is walked in longer chunks than alone.
Its values do not depend on the chunks (each row is the same arithmetic on the
same window of three planes), only the order of the dot products does: the
operator and the V-cycle have to be equal bit for bit, solves to rounding.  The
part alone is compared with the oracle.

Tolerances: operator rows sum fewer than 700 products, 8e-14 relative in any
order; 100 roundings of 2^-53 elementwise on either side where magnitudes vary;
PCG to 1e-10 from dot products that differ by 1e-15 at most."""
import numpy as np
import pytest

from gmgs import Solver, synthetic
from gmgs_oracle import Oracle, Params

pytestmark = pytest.mark.gpu

LEVELS = 3
NZ = 33                                             # padded to 36: 37 planes of nodes
# edge of the box in elements, by the planes per chunk it gives on 152 SMs; the last chunk is short in each
BOXES = {"2 planes": 95, "3 planes": 239, "5 planes": 335, "13 planes": 543, "32 planes": 895}


def part(ny, nx, seed=3):
    """A block with voids, and a notch: from the second tile column on the planes 13..19 are empty."""
    vox = synthetic.sphere_voids(nx, ny, NZ, 2 if min(nx, ny) >= 30 else 0, seed)
    vox[:, 14:, 12:20] = 0
    return np.asfortranarray(vox)


def handles(vox, box, rho=None):
    ny, nx, nz = vox.shape
    out = []
    for edge in (None, box):
        v = vox
        if edge is not None:
            v = np.zeros((edge, edge, nz), dtype=vox.dtype, order="F")
            v[:ny, :nx] = vox
        s = Solver(v, omega=0.4, num_levels=LEVELS)
        s.set_bc(*synthetic.boundary_conditions(vox, LEVELS))
        s.set_tolerance(1e-10, 400)
        if rho is not None:
            s.set_density(rho, 3.0)
        out.append(s)
    return out


def field(kind, vox, seed=5):
    """(z, x, y) values on the compact nodes, as an interleaved vector, and the nodes' plane numbers."""
    mask = synthetic.solid_node_mask(vox)
    iz = np.broadcast_to(np.arange(mask.shape[2]), mask.shape).ravel(order="F")[mask.ravel(order="F")]
    x = np.random.default_rng(seed).standard_normal((len(iz), 3))
    if kind == "ranges":        # planes near each other and far apart: the stages change inside a chunk
        power = np.array([0, 0, 0, 0, 40, 40, 40, 40, 0, 0, 8, 8, 16, 16, 24, 24, 32, 32, 0, 0, 0, 300, 300, 300, 300, 300,
                          0, 0, 0, 0, 10, 20, 30, 40])
        x *= np.exp2(-power[iz].astype(float))[:, None]
        x[iz == 29] = 0
    if kind == "nan":
        x[np.flatnonzero(iz == 6)[40], 1] = np.nan
        x[np.flatnonzero(iz == 24)[50], 0] = np.inf
    return x.reshape(-1)


@pytest.mark.parametrize("density", [False, True], ids=["uniform", "density"])
@pytest.mark.parametrize("box", BOXES)
@pytest.mark.parametrize("ny,nx", [(33, 31), (30, 32)], ids=["34x32 nodes", "31x33 nodes"])
def test_walks_agree(ny, nx, box, density):
    if box == "32 planes" and (density or ny == 30):
        pytest.skip("once: the box is 29M slots")
    vox = part(ny, nx)
    rho = synthetic.density(int(vox.sum()), (0.2, 1.0), 8) if density else None
    alone, boxed = handles(vox, BOXES[box], rho)
    for kind in ("plain", "ranges", "nan"):
        x = field(kind, vox)
        a, b = alone.apply_operator(x), boxed.apply_operator(x)
        assert np.array_equal(a, b, equal_nan=True), kind
        assert np.array_equal(alone.apply_preconditioner(x), boxed.apply_preconditioner(x), equal_nan=True), kind
    ua, ub = alone.solve(), boxed.solve()
    assert alone.iterations == boxed.iterations
    assert np.linalg.norm(ua - ub) <= 1e-9 * np.linalg.norm(ua)


@pytest.mark.parametrize("density", [False, True], ids=["uniform", "density"])
@pytest.mark.parametrize("ny,nx", [(14, 14), (15, 15), (16, 16), (14, 16), (16, 15), (30, 31), (31, 30), (32, 32)])
def test_extents_around_the_tile(ny, nx, density):
    """15, 16, 17 and 31, 32, 33 nodes along either side of the 16 x 16 tile, against the oracle."""
    vox = part(ny, nx)
    o = Oracle(vox, Params(omega=0.4, num_levels=LEVELS))
    o.apply_boundary_condition(*synthetic.boundary_conditions(vox, LEVELS))
    rho = synthetic.density(int(vox.sum()), (0.2, 1.0), 8) if density else None
    if density:
        o.set_density(rho, 3.0)
    o.setup()
    _, s = handles(vox, 95, rho)
    lv = o.levels[0]
    x = field("plain", vox)
    y = s.apply_operator(x)
    assert np.linalg.norm(y - o.atx(x, 0)) <= 2e-13 * np.linalg.norm(y)
    x = field("ranges", vox)
    size = np.abs(x[lv.eDofMat]) @ np.abs(lv.Ks) * (1.0 if lv.eleScale is None else lv.eleScale[:, None])
    bound = np.zeros(lv.numDOFs)
    np.add.at(bound, lv.eDofMat.ravel(), size.ravel())      # sum over the elements of |Ke| |x|
    assert np.all(np.abs(s.apply_operator(x) - o.atx(x, 0)) <= 2 * 100 * 2.0 ** -53 * bound)
    r = field("plain", vox)
    r[lv.fixedDOFs] = 0
    z = o.vcycle(r)
    assert np.linalg.norm(s.apply_preconditioner(r) - z) <= 1e-10 * np.linalg.norm(z)
