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


# The stages of the factorised stencil run on 96-bit integers where the values of
# a window stay within 2^23 of each other, on FP64 elsewhere.  Elementwise bound:
# every row's terms are rounded at most 100 times at 2^-53 (FP64 stages, 3 x 3 x 3
# weights on three components in sequence), so |y - K x| <= 100 * 2^-53 |K| |x|.
@pytest.mark.parametrize("spread", [0, 10, 22, 24, 60, 200], ids=lambda s: f"2^{s}")
@pytest.mark.parametrize("scale", [1.0, 1e-200, 1e-290, 1e250])
def test_operator_elementwise_over_dynamic_ranges(spread, scale):
    import scipy.sparse as sp
    o, s = pair((18, 17, 12), 1, 2, (1.0, 1.0, 1.0), None, 9)
    o.setup()
    K = sp.csr_matrix(o.assemble_level(0))
    rng = np.random.default_rng(spread)
    n = o.levels[0].numDOFs
    x = rng.choice([-1.0, 1.0], n) * np.repeat(np.exp2(rng.uniform(-spread, 0, n // 3)), 3) * rng.uniform(0.5, 1, n) * scale
    free = np.ones(n, bool)
    free[o.levels[0].fixedDOFs] = False
    with np.errstate(under="ignore"):
        err, bound = np.abs(s.apply_operator(x, 1) - K @ x), 100 * 2.0 ** -53 * (abs(K) @ abs(x))
    assert np.all(err[free] <= 2 * bound[free] + 1e-322)     # the reference product rounds as well


@pytest.mark.parametrize("ele", [(1.0, 1.0, 30.0), (1.0, 40.0, 1.0), (0.02, 1.0, 1.0), (1.0, 6.0, 0.5)])
def test_operator_on_flat_voxels(ele):
    """Coefficients far apart: within 2^11 of each other on integers, beyond on FP64."""
    o, s = pair((18, 17, 12), 1, 2, ele, None, 9)
    o.setup()
    x = np.random.default_rng(1).standard_normal(o.levels[0].numDOFs)
    assert rel(s.apply_operator(x, 1), o.atx(x, 0)) < TOL


@pytest.mark.parametrize("bad", [np.nan, np.inf, -np.inf])
def test_operator_keeps_non_finite_values(bad):
    """A NaN or infinity reaches the rows coupled to it and no others."""
    o, s = pair((18, 17, 20), 0, 2, (1.0, 1.0, 1.0), None, 9)
    o.setup()
    n = o.levels[0].numDOFs
    x = np.random.default_rng(1).standard_normal(n)
    clean = s.apply_operator(x, 1)
    at = 3 * (19 * 18 * 10 + 19 * 8 + 9)          # an interior node
    x[at] = bad
    y = s.apply_operator(x, 1)
    node = np.arange(n // 3)
    iy, ix, iz = node % 19, node // 19 % 18, node // (19 * 18)
    near = (abs(iy - iy[at // 3]) <= 1) & (abs(ix - ix[at // 3]) <= 1) & (abs(iz - iz[at // 3]) <= 1)
    assert not np.isfinite(y.reshape(-1, 3)[near]).all(axis=1).any()
    assert np.all(np.abs(y - clean).reshape(-1, 3)[~near] <= 1e-13)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_later_densities_equal_a_fresh_handle(precision):
    """The second density of a handle reuses the hierarchy of the first; device and
    host densities give the same bits, and what was refused is refused."""
    torch = pytest.importorskip("torch")
    from gmgs import GMGSError
    from gmgs.autograd import compliance
    vox = synthetic.sphere_voids(20, 18, 28, 2, 6)
    fixed, loads = synthetic.boundary_conditions(vox, 3)
    first, second = (synthetic.density(int(vox.sum()), (0.2, 1.0), k) for k in (1, 2))

    def handle():
        s = Solver(vox, omega=0.4, num_levels=3, precision=precision)
        s.set_bc(fixed, loads)
        return s

    fresh, kept = handle(), handle()
    fresh.set_density(second, 2.0)
    u_ref, g_ref = fresh.solve(), fresh.grad()
    kept.set_density(first, 3.0)
    kept.solve()
    kept.set_bc(fixed, loads)
    with pytest.raises(GMGSError):
        kept.set_density(np.where(np.arange(len(second)) == 7, -1.0, second), 2.0)
    on_gpu = torch.tensor(second, device="cuda")
    torch.cuda.synchronize()
    kept.set_density_dev(on_gpu.data_ptr(), 2.0)
    u = kept.solve()
    assert np.array_equal(u, u_ref) and np.array_equal(kept.grad(), g_ref)
    assert abs(kept.load_work() - kept.load_vector() @ u) <= 1e-12 * abs(kept.load_work())
    for bad in (np.nan, np.inf, 0.0):
        wrong = on_gpu.clone()
        wrong[3] = bad
        torch.cuda.synchronize()
        with pytest.raises(GMGSError):
            kept.set_density_dev(wrong.data_ptr(), 2.0)
    for device in ("cpu", "cuda"):
        rho = torch.tensor(second, device=device, requires_grad=True)
        j = compliance(rho, kept, 2.0)
        (2 * j).backward()
        assert abs(j.item() - kept.load_vector() @ u_ref) <= 1e-12 * abs(j.item())
        assert np.array_equal(rho.grad.cpu().numpy(), 2 * g_ref)


# The transfers sum as 64-bit integers on the exponent of the largest value, in
# FP64 for zeros, non-finite values and near the ends of the range.
def vcycle_inputs():
    o, s = pair((20, 18, 26), 3, 3, (1.0, 1.0, 1.0), None, 5)
    r = np.random.default_rng(8).standard_normal(o.levels[0].numDOFs)
    r[o.levels[0].fixedDOFs] = 0
    return o, s, r


@pytest.mark.parametrize("power", [-600, -40, 40, 600])
def test_vcycle_scales_by_powers_of_two(power):
    """All steps are linear, and exact in a power of two while nothing leaves the range."""
    o, s, r = vcycle_inputs()
    assert np.array_equal(s.apply_preconditioner(np.ldexp(r, power)), np.ldexp(s.apply_preconditioner(r), power))


@pytest.mark.parametrize("spread", [0, 6, 8, 30, 52, 70, 300], ids=lambda s: f"2^{s}")
def test_vcycle_over_dynamic_ranges(spread):
    o, s, r = vcycle_inputs()
    o.setup()
    r *= np.exp2(np.random.default_rng(spread).uniform(-spread, 0, r.size))
    r[::7] = 0
    assert rel(s.apply_preconditioner(r), o.vcycle(r)) < 1e-10


@pytest.mark.parametrize("bad", [np.nan, np.inf, -np.inf])
def test_vcycle_keeps_non_finite_values(bad):
    o, s, r = vcycle_inputs()
    assert np.array_equal(s.apply_preconditioner(0.0 * r), 0.0 * r)
    at = np.flatnonzero(r)[r.size // 2]
    r[at] = bad
    z = s.apply_preconditioner(r)
    assert not np.isfinite(z[at]) and np.isnan(z).any()
