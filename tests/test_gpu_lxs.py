"""The triple kernels of L and L* (ddc_lxs.cu) at the edges of their chunks:
spheres without neighbours, with a handful of triples, around one chunk and
over several, for role counts of every kind (lmax 0 to 12).  FP64 against the
oracle's lx / lstarx (matvec.f90:94-235); the FP32 operators of the mixed
contexts against the same.

Tolerances (2-norm over the vector, relative): FP64 1e-13 as elsewhere; FP32
64 * 2^-24 = 3.8e-6: geometry, powers, recurrence, contraction and gather
round a value some tens of times at 2^-24 each."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _spheres(kind, seed):
    from ddpcm_b200 import molecules as M
    if kind == "pair":  # a touching pair, a deep overlap and a lone sphere
        return dict(x=np.array([0.0, 5.9, 20.0, 21.0, 60.0]), y=np.array([0.0, 0.0, 0.0, 0.5, 0.0]),
                    z=np.array([0.0, 0.0, 0.0, 0.0, 0.0]), r=np.array([3.0, 3.0, 3.0, 2.6, 2.0]))
    return M.to_bohr(M.make_molecule(40 if kind == "small" else 70, seed))


@pytest.mark.parametrize("kind,ngrid", [("pair", 110), ("small", 110), ("large", 434)])
@pytest.mark.parametrize("lmax", [0, 2, 4, 5, 6, 7, 8, 9, 10, 12])
def test_operators_at_chunk_edges(oracle, kind, ngrid, lmax):
    from ddpcm_b200.ddcosmo import DDCosmo, PREC_FP64, PREC_MIXED
    m = _spheres(kind, 500 + lmax)
    n, nylm = len(m["r"]), (lmax + 1) ** 2
    rng = np.random.default_rng(lmax)
    x, s = rng.normal(size=(2, n, nylm))
    ref = oracle.RefDD(lmax, ngrid, 10, 1, 78.3553, 0.1).init(m["x"], m["y"], m["z"], m["r"])
    want = ref.lx(x), ref.lstarx(s)
    for prec, tol in ((PREC_FP64, 1e-13), (PREC_MIXED, 64 * 2.0 ** -24)):
        with DDCosmo(lmax=lmax, ngrid=ngrid, iconv=10, eta=0.1, precision=prec) as dd:
            dd.ddinit(m["x"], m["y"], m["z"], m["r"])
            pair = dd.lx_lstarx(x, s)
            alone = dd.lx(x), dd.lstarx(s)
        for got in (pair, alone):
            for a, b in zip(got, want):
                assert np.linalg.norm(a - b) <= tol * np.linalg.norm(b)
        if kind == "pair":  # the lone sphere has no triples
            assert np.all(pair[0][-1] == 0.0) and np.all(pair[1][-1] == 0.0)


@pytest.mark.parametrize("n", [296, 297])
@pytest.mark.parametrize("lmax", [0, 1, 3, 4, 5, 6, 7, 8, 9, 10, 11, 12])
def test_both_operators_by_halves_and_together(oracle, n, lmax):
    """lx and lstarx in one launch: by blocks of their own up to 296 spheres,
    from one pass over the triples beyond."""
    from ddpcm_b200 import molecules as M
    from ddpcm_b200.ddcosmo import DDCosmo, PREC_FP64, PREC_MIXED
    m = M.to_bohr(M.make_molecule(n, 700 + lmax))
    rng = np.random.default_rng(lmax)
    x, s = rng.normal(size=(2, n, (lmax + 1) ** 2))
    ref = oracle.RefDD(lmax, 110, 10, 1, 78.3553, 0.1).init(m["x"], m["y"], m["z"], m["r"])
    want = ref.lx(x), ref.lstarx(s)
    for prec, tol in ((PREC_FP64, 1e-13), (PREC_MIXED, 64 * 2.0 ** -24)):
        with DDCosmo(lmax=lmax, ngrid=110, iconv=10, eta=0.1, precision=prec) as dd:
            dd.ddinit(m["x"], m["y"], m["z"], m["r"])
            for got, w in zip(dd.lx_lstarx(x, s), want):
                assert np.linalg.norm(got - w) <= tol * np.linalg.norm(w)


@pytest.mark.parametrize("n,lmax,ngrid", [
    # all folded (ddc_fold.cu: eight spheres per block); the other paths of the
    # mixed operators are held in test_gpu_tcgen05.py
    (9, 8, 110),      # one sphere in the last block
    (1603, 8, 110),   # three, of many blocks
    (1190, 10, 110),  # fewer points than harmonics
    (14305, 2, 26)])  # few harmonics, a class of them without any
def test_contractions_by_shape(oracle, n, lmax, ngrid):
    """The projection and expansion GEMMs of every dispatch branch (remainders
    in all three dimensions), through lx and lstarx."""
    from ddpcm_b200 import molecules as M
    from ddpcm_b200.ddcosmo import DDCosmo, PREC_FP64, PREC_MIXED
    m = M.to_bohr(M.make_molecule(n, 900))
    rng = np.random.default_rng(n)
    x, s = rng.normal(size=(2, n, (lmax + 1) ** 2))
    ref = oracle.RefDD(lmax, ngrid, 10, 1, 78.3553, 0.1).init(m["x"], m["y"], m["z"], m["r"])
    want = ref.lx(x), ref.lstarx(s)
    for prec, tol in ((PREC_FP64, 1e-13), (PREC_MIXED, 64 * 2.0 ** -24)):
        with DDCosmo(lmax=lmax, ngrid=ngrid, iconv=10, eta=0.1, precision=prec) as dd:
            dd.ddinit(m["x"], m["y"], m["z"], m["r"])
            for a, b in zip(dd.lx_lstarx(x, s), want):
                assert np.linalg.norm(a - b) <= tol * np.linalg.norm(b)
