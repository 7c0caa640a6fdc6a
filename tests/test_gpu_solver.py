"""The device Jacobi/DIIS (ddc_solver.cu) at the edges of its chunks (512,
2,048 and 8,192 elements) and of its history (no DIIS, the shortest and the
longest history the parameters allow), one system alone and both together,
FP64 and mixed.  The stop test bounds the H-norm of the Jacobi increment of
the last extrapolation, so the increment of the returned solution itself,
formed here with the FP64 operator, is of that size: at most 10 times the
tolerance (the increment changes by the contraction of one iteration)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _increment(dd, x, g, op):
    return dd.hnorm(dd.ldm1x(g - op(x)) - x)


@pytest.mark.parametrize("n,lmax,ngrid,kw", [
    (1, 0, 26, {}), (3, 2, 26, {}), (11, 6, 110, {}), (21, 6, 110, dict(ndiis=11)),
    (42, 6, 110, dict(ndiis=32)), (60, 6, 110, dict(ndiis=0, max_iter=2000)),
    (113, 8, 110, dict(pair_solves=0)), (5003, 10, 302, {}), (5011, 10, 302, {}),
    (10021, 10, 302, {}), (10021, 10, 302, dict(ndiis=11))])
@pytest.mark.parametrize("prec", [0, 1])
def test_solution_meets_the_stop_test(n, lmax, ngrid, kw, prec):
    from ddpcm_b200 import molecules as M
    from ddpcm_b200.ddcosmo import DDCosmo
    m = M.to_bohr(M.make_molecule(n, 40 + n))
    p = dict(lmax=lmax, ngrid=ngrid, iconv=10, eta=0.1)
    with DDCosmo(precision=prec, **p, **kw) as dd:
        out = dd.energy_forces(m["q"], m["x"], m["y"], m["z"], m["r"])
    with DDCosmo(**p) as dd:
        dd.ddinit(m["x"], m["y"], m["z"], m["r"])
        phi, psi = dd.mkrhs(m["q"], m["x"], m["y"], m["z"])
        g = dd.rhs(phi)
        assert _increment(dd, out["sigma"], g, dd.lx) <= 1e-9
        assert _increment(dd, out["s"], psi, dd.lstarx) <= 1e-9
    for side in ("direct", "adjoint"):
        i = out["info"][side]
        assert i["converged"] and i["iterations"] >= 1
        norms = i["norms"]
        assert len(norms) == min(i["iterations"], 256) and all(v > 0.0 for v in norms[:-1])
        if prec == 0 and i["iterations"] <= 256:
            assert norms[-1] < 1e-10 and norms[-1] == i["final_norm"]


def test_budget_runs_out():
    from ddpcm_b200 import molecules as M
    from ddpcm_b200.ddcosmo import DDCosmo, DDCosmoError, DDC_ERR_NOCONV
    m = M.to_bohr(M.make_molecule(100, 3))
    for prec in (0, 1):
        with DDCosmo(lmax=6, ngrid=110, iconv=10, eta=0.1, precision=prec, max_iter=5) as dd:
            with pytest.raises(DDCosmoError) as e:
                dd.energy_forces(m["q"], m["x"], m["y"], m["z"], m["r"])
            assert e.value.status == DDC_ERR_NOCONV


@pytest.mark.parametrize("prec", [0, 1])
@pytest.mark.parametrize("n", [3092, 3093, 3135, 3136])
def test_where_the_chunks_grow(n, prec):
    """49 elements per sphere: 151,508 elements by 512 and 151,557 by 2,048, the
    last chunk with 5 elements (k_extrap's other three blocks of it have none);
    75 chunks and 15 elements, 64 more."""
    test_solution_meets_the_stop_test(n, 6, 110, {}, prec)


def test_no_early_stop():
    """Small molecules to 1e-12: the coefficients of the late extrapolations
    must not be rounding noise, which stops some solves with errors of 1e-10 to
    3e-9.  With exact coefficients the largest error of 40 molecules is 7e-12
    of a solution of norm about 1; the increment of the returned solution
    stays within 50 times the tolerance."""
    from ddpcm_b200 import molecules as M
    from ddpcm_b200.ddcosmo import DDCosmo
    with DDCosmo(lmax=6, ngrid=110, iconv=12, eta=0.1) as dd:
        for seed in range(20, 50):
            m = M.to_bohr(M.make_molecule(12, seed, globule=False))
            out = dd.energy_forces(m["q"], m["x"], m["y"], m["z"], m["r"])
            dd.ddinit(m["x"], m["y"], m["z"], m["r"])
            phi, psi = dd.mkrhs(m["q"], m["x"], m["y"], m["z"])
            assert _increment(dd, out["sigma"], dd.rhs(phi), dd.lx) <= 5e-11
            assert _increment(dd, out["s"], psi, dd.lstarx) <= 5e-11
