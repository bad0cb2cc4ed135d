"""Stiffnesses near the end of the exponent range: subnormal pivots of the coarsest
level are positive and stay accepted as long as their inverse is finite.

The matrix of E = 2^-k is that of E = 1 times 2^-k up to multiples of 2^-1074 (the
smallest entries lie above 2^-1030, so 2^-45 of them at most); U scales
with 2^k.  Tolerance: 2^-45 times a condition number below 2^12, and PCG to
1e-10."""
import numpy as np
import pytest

from gmgs import Solver, synthetic
from gmgs_oracle import Oracle, Params

pytestmark = pytest.mark.gpu


def test_subnormal_pivots():
    vox = synthetic.sphere_voids(4, 4, 4, 0, 1)
    fixed, loads = synthetic.boundary_conditions(vox, 2)
    o = Oracle(vox, Params(omega=0.4, num_levels=2))
    o.apply_boundary_condition(fixed, loads)
    o.setup()
    lv = o.levels[-1]
    K = o.assemble_level(1)[np.ix_(lv.freeDOFs, lv.freeDOFs)]
    pivot, inverse = (np.diag(np.linalg.cholesky(K)) ** 2).min(), np.abs(np.linalg.inv(K)).max()
    k = 1022 + int(np.ceil(np.log2(pivot)))             # the smallest pivot falls below 2^-1022
    assert pivot * 2.0 ** -k < 2.0 ** -1022 and np.log2(inverse) + k < 1023.5

    def solve(k):
        s = Solver(vox, omega=0.4, num_levels=2, youngs_modulus=2.0 ** -k)
        scaled, shift = loads.copy(), 2 * k // 5       # keeps the dot products of r and of U in range
        scaled[:, 1:] *= 2.0 ** -shift
        s.set_bc(fixed, scaled)
        s.set_tolerance(1e-10, 200)
        return np.ldexp(s.solve(), -(k - shift))

    u = solve(0)
    assert np.linalg.norm(solve(k) - u) <= 2e-9 * np.linalg.norm(u)
