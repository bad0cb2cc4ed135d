"""Where the FP64 operator may use its integer stages (fine64.cu): rows whose
components lie far apart, and subnormal patches beside normal values.

The reference is the interior stencil of the box element as sums of products of
the 1-D operators m = [1 4 1], k = [-1 2 -1], d = [-1 0 1], with exact zeros
where two components do not couple (an assembled matrix has rounding noise
there).  Elementwise bound as in test_gpu_fine64.py: a row's terms are rounded at
most 100 times at 2^-53, on either side, so |y - K x| <= 2 * 100 * 2^-53 |K| |x|."""
import itertools

import numpy as np
import pytest

from gmgs import Solver, synthetic

pytestmark = pytest.mark.gpu

NU = 0.3
BOUND = 2 * 100 * 2.0 ** -53
M1, K1, D1 = (np.array(v, float) for v in ([1, 4, 1], [-1, 2, -1], [-1, 0, 1]))


def stencil(ele):
    """S[c, b] over the offsets (z, x, y), the physical y axis against the index."""
    x, y, z = ele
    lam, mu = NU / ((1 + NU) * (1 - 2 * NU)), 0.5 / (1 + NU)
    S = np.zeros((3, 3, 3, 3, 3))

    def tensor(fz, fx, fy):
        return np.einsum("i,j,k->ijk", fz, fx, fy)

    for c in range(3):
        e = [lam + 2 * mu if c == a else mu for a in range(3)]
        S[c, c] = (e[0] * y * z / (36 * x) * tensor(M1, K1, M1) + e[1] * x * z / (36 * y) * tensor(M1, M1, K1)
                   + e[2] * x * y / (36 * z) * tensor(K1, M1, M1))
    g = (lam + mu) / 24
    S[0, 1] = S[1, 0] = g * z * tensor(M1, D1, D1)
    S[0, 2] = S[2, 0] = -g * y * tensor(D1, D1, M1)
    S[1, 2] = S[2, 1] = g * x * tensor(D1, M1, D1)
    return S


def apply_interior(S, u):
    """Rows of the interior nodes: u (3, z, x, y) -> (3, z - 2, x - 2, y - 2), in the widest float numpy has."""
    u = u.astype(np.longdouble)
    nz, nx, ny = (n - 2 for n in u.shape[1:])
    y = np.zeros((3, nz, nx, ny), np.longdouble)
    for c, b in itertools.product(range(3), range(3)):
        for o in itertools.product(range(3), repeat=3):
            if S[c, b][o]:
                y[c] += S[c, b][o] * u[b, o[0]:o[0] + nz, o[1]:o[1] + nx, o[2]:o[2] + ny]
    return y


NY, NX, NZ = 18, 17, 12


def block(ele=(1.0, 1.0, 1.0)):
    vox = synthetic.sphere_voids(NX, NY, NZ, 0, 1)
    fixed, loads = synthetic.boundary_conditions(vox, 2)
    s = Solver(vox, ele_size=ele, poisson_ratio=NU, omega=0.4, num_levels=2)
    s.set_bc(fixed, loads)
    return s


def check(s, S, u, floor=0.0):
    x = u.transpose(1, 2, 3, 0).reshape(-1)             # compact order: y fastest, then x, z; components interleaved
    y = s.apply_operator(np.ascontiguousarray(x)).reshape(NZ + 1, NX + 1, NY + 1, 3).transpose(3, 0, 1, 2)[:, 1:-1, 1:-1, 1:-1]
    err = np.abs(y - apply_interior(S, u))
    bound = BOUND * apply_interior(abs(S), abs(u))
    assert np.all(err <= bound + floor), f"{int((err > bound + floor).sum())} rows off, worst {float((err - bound).max()):.3g} beyond"


# the large components where they do not couple into the small one's row (the
# node itself, its face neighbours) or only some of them do
PLACES = {"same node": (0, 0, 0), "x face": (0, 1, 0), "y face": (0, 0, 1), "z face": (1, 0, 0), "xy edge": (0, 1, 1),
          "xz edge": (1, 1, 0), "yz edge": (1, 0, 1), "corner": (1, 1, 1), "apart": (0, 3, 2)}


@pytest.mark.parametrize("ele", [(1.0, 1.0, 1.0), (0.05, 1.0, 1.0), (1.0, 1.0, 20.0)], ids=["cube", "flat x", "long z"])
@pytest.mark.parametrize("place", PLACES)
def test_components_far_apart(place, ele):
    s, S = block(ele), stencil(ele)
    dz, dx, dy = PLACES[place]
    for small, large in itertools.permutations(range(3), 2):
        for k in (0, 12, 19, 22, 26, 30, 40, 50, 60, 70, 90, 300):
            u = np.zeros((3, NZ + 1, NX + 1, NY + 1))
            u[small, 6, 7, 8] = 0.8 * 2.0 ** -k
            u[large, 6 + dz, 7 + dx, 8 + dy] = 0.9
            u[large, 6 - dz, 7 - dx, 8 - dy] = 0.7
            check(s, S, u)


@pytest.mark.parametrize("component", [0, 1, 2])
def test_component_that_is_noise_on_a_plane_or_everywhere(component):
    """A symmetry plane, and an axial field: a component at rounding level there."""
    s, S = block(), stencil((1.0, 1.0, 1.0))
    rng = np.random.default_rng(component)
    for where in (np.s_[component, :, 8, :], np.s_[component, :, :, 9], np.s_[component, 5], np.s_[component]):
        u = rng.uniform(0.5, 1, (3, NZ + 1, NX + 1, NY + 1)) * rng.choice([-1.0, 1.0], (3, NZ + 1, NX + 1, NY + 1))
        u[where] *= 2.0 ** -54
        check(s, S, u)
        u[[c for c in range(3) if c != component]] = 0.25     # no differences left in the others
        check(s, S, u)


# A row of subnormal values: every product and sum may round to a multiple of
# 2^-1074, at most 100 times on either side.
def test_subnormal_patch_beside_normal_values():
    s, S = block(), stencil((1.0, 1.0, 1.0))
    rng = np.random.default_rng(4)
    u = np.zeros((3, NZ + 1, NX + 1, NY + 1))
    u[:, :, :6, :] = rng.uniform(0.5, 1, u[:, :, :6, :].shape)
    u[:, :, 9:14, 4:12] = rng.uniform(0.5, 1, (3, NZ + 1, 5, 8)) * 2.0 ** -1024
    y = apply_interior(S, u)
    assert np.abs(y[:, 2, 10, 6]).max() > 1e6 * 200 * 2.0 ** -1074
    check(s, S, u, floor=200 * 2.0 ** -1074)
