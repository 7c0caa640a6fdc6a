"""Small FP64 solves to 1e-12 against direct solutions of the same equations:
(1 / facl + L) x = g with L assembled column by column from lx and lstarx.

At the stop the H-norm of the increment per sphere is below 1e-12, so its 2-norm
is at most sqrt(n (1 + lmax)) 1e-12 = 9.2e-12 for 12 spheres at lmax 6; the
error is that over one less the contraction of an iteration, at most 0.9 for
these chains: 9.2e-11 of a solution of norm about 1.  Extrapolation
coefficients that are rounding noise stop one solve in five with an error of
1e-10 to 3e-8 instead."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("seed", range(100, 124))
def test_chain_against_direct_solution(seed):
    from ddpcm_b200 import molecules as M
    from ddpcm_b200.ddcosmo import DDCosmo
    n, lmax = 12, 6
    m = M.to_bohr(M.make_molecule(n, seed, globule=False))
    with DDCosmo(lmax=lmax, ngrid=110, iconv=12, eta=0.1) as dd:
        out = dd.energy_forces(*(m[k] for k in "qxyzr"))
        phi, psi = dd.mkrhs(m["q"], m["x"], m["y"], m["z"])
        g = dd.rhs(phi)
        unit = np.eye(n * (lmax + 1) ** 2).reshape(-1, n, (lmax + 1) ** 2)
        lx, ls = (np.stack([op(u).ravel() for u in unit], 1) for op in (dd.lx, dd.lstarx))
    facl = np.repeat((2 * np.arange(lmax + 1) + 1) / (4 * np.pi), 2 * np.arange(lmax + 1) + 1)
    diag = np.diag(np.tile(1.0 / facl, n))
    for got, op, rhs in ((out["sigma"], lx, g), (out["s"], ls, psi)):
        want = np.linalg.solve(diag + op, rhs.ravel())
        assert np.linalg.norm(got.ravel() - want) <= 1e-10 * np.linalg.norm(want)
