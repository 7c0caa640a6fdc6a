"""The folded contractions (ddc_fold.cu) over the grid's orbits and the eight
classes of harmonics: classes without harmonics (lmax 0 and 1), of one to four
row tiles, grids whose orbits fit one pass and grids that need two (770 points:
109 orbits, 974: 136, 1202: 166; 96 per pass), a last block of one sphere.
Through lx and lstarx (matvec.f90:94-235) against the oracle; tolerances as in
test_gpu_lxs.py (FP64 1e-13, FP32 fields 64 * 2^-24)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lmax,ngrid", [(0, 6), (1, 14), (2, 38), (4, 50), (5, 86), (7, 194),
                                        (9, 590), (11, 350), (12, 770), (8, 974), (12, 1202)])
@pytest.mark.parametrize("n", [8, 17])
def test_operators_by_orbits_and_classes(oracle, lmax, ngrid, n):
    from ddpcm_b200 import molecules as M
    from ddpcm_b200.ddcosmo import DDCosmo, PREC_FP64, PREC_MIXED
    m = M.to_bohr(M.make_molecule(n, 300 + lmax))
    rng = np.random.default_rng(ngrid)
    x, s = rng.normal(size=(2, n, (lmax + 1) ** 2))
    ref = oracle.RefDD(lmax, ngrid, 10, 1, 78.3553, 0.1).init(m["x"], m["y"], m["z"], m["r"])
    want = ref.lx(x), ref.lstarx(s)
    for prec, tol in ((PREC_FP64, 1e-13), (PREC_MIXED, 64 * 2.0 ** -24)):
        with DDCosmo(lmax=lmax, ngrid=ngrid, iconv=10, eta=0.1, precision=prec) as dd:
            assert dd.ddinit(m["x"], m["y"], m["z"], m["r"]).ngrid == ngrid
            for got, w in zip(dd.lx_lstarx(x, s), want):
                assert np.linalg.norm(got - w) <= tol * np.linalg.norm(w)
