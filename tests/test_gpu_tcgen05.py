"""The mixed operators' contractions on tcgen05 (ddc_tc.cu) below the size from
which a solve takes them (DDC_FOLD=0), the folded ones (ddc_fold.cu) and the
FP32 SIMT ones (DDC_TC_OFF=1), each against the FP64 oracle's lx and lstarx
(matvec.f90:94, :161), and the choice between them on both sides of 2e8
products of harmonics and points.  Which path ran shows in the bits: all three
are deterministic and round differently.

Bars as in test_gpu_tc.py: 1e-5 of the largest entry, and three times the SIMT
error (a product of the three-term TF32 split carries 2^-21 against 2^-24)."""
import contextlib
import os

import numpy as np
import pytest

from conftest import load_golden

pytestmark = pytest.mark.gpu

BAR = 1e-5


@contextlib.contextmanager
def _environment(**kw):
    os.environ.update(kw)
    try:
        yield
    finally:
        for k in kw:
            os.environ.pop(k)


def _apply(m, lmax, ngrid, x, s, **env):
    from ddpcm_b200.ddcosmo import PREC_MIXED, DDCosmo
    with _environment(**env), DDCosmo(lmax=lmax, ngrid=ngrid, iconv=10, eta=0.1,
                                      precision=PREC_MIXED) as dd:
        dd.ddinit(m["x"], m["y"], m["z"], m["r"])
        return [*dd.lx_lstarx(x, s), dd.lx(x), dd.lstarx(s)]


def _case(oracle, m, lmax, ngrid, seed):
    rng = np.random.default_rng(seed)
    d = oracle.RefDD(lmax, ngrid, 10, 1, 78.3553, 0.1).init(m["x"], m["y"], m["z"], m["r"])
    x, s = rng.standard_normal((2, d.nsph, d.nylm))
    y, z = d.lx(x), d.lstarx(s)
    return x, s, [y, z, y, z]


def _errors(got, want):
    return [np.abs(a - b).max() / np.abs(b).max() for a, b in zip(got, want)]


def _differ(a, b):
    return all(not np.array_equal(u, v) for u, v in zip(a, b))


def _globule(n):
    from ddpcm_b200 import molecules as M
    return M.to_bohr(M.make_molecule(n, n))


@pytest.mark.parametrize("lmax,ngrid,mol", [
    (0, 110, "caffeine"), (6, 302, "crambin"), (8, 302, "taxol"), (10, 590, "crambin"),
    (6, 302, 2400), (6, 302, 9472), (9, 434, 161), (4, 50, 33)])
def test_tcgen05_below_the_line(oracle, lmax, ngrid, mol):
    """One to four 32-wide k-chunks of the expansion, one to five 128-row grid
    tiles, grids that are no multiple of four points (rows padded for TMA), one
    tile and many, a last tile of one sphere."""
    m = load_golden(mol)["mol"] if isinstance(mol, str) else _globule(mol)
    x, s, want = _case(oracle, m, lmax, ngrid, 100 + lmax)
    tc = _apply(m, lmax, ngrid, x, s, DDC_FOLD="0")
    simt = _apply(m, lmax, ngrid, x, s, DDC_TC_OFF="1")
    fold = _apply(m, lmax, ngrid, x, s)
    for a, b in ((tc, simt), (tc, fold), (simt, fold)):
        assert _differ(a, b)
    for et, es, ef in zip(_errors(tc, want), _errors(simt, want), _errors(fold, want)):
        assert max(et, ef) <= BAR
        assert et <= 3.0 * es + 1e-7


@pytest.mark.parametrize("n,lmax,ngrid", [(13515, 6, 302), (2800, 10, 590), (2353, 11, 590)])
def test_folded_up_to_the_line(oracle, n, lmax, ngrid):
    m = _globule(n)
    assert n * (lmax + 1) ** 2 * ngrid <= 200_000_000
    x, s, want = _case(oracle, m, lmax, ngrid, n)
    got = _apply(m, lmax, ngrid, x, s)
    assert max(_errors(got, want)) <= BAR
    for a, b in zip(got, _apply(m, lmax, ngrid, x, s, DDC_FOLD="1")):
        assert np.array_equal(a, b)
    assert _differ(got, _apply(m, lmax, ngrid, x, s, DDC_FOLD="0"))


@pytest.mark.parametrize("n,lmax,ngrid", [(13537, 6, 302), (2817, 10, 590), (2371, 11, 590)])
def test_beyond_the_line(oracle, n, lmax, ngrid):
    """tcgen05 up to 128 harmonics, SIMT for more; a last tile of one sphere."""
    m = _globule(n)
    assert n * (lmax + 1) ** 2 * ngrid > 200_000_000
    x, s, want = _case(oracle, m, lmax, ngrid, n)
    got = _apply(m, lmax, ngrid, x, s)
    simt = _apply(m, lmax, ngrid, x, s, DDC_TC_OFF="1")
    assert _differ(got, _apply(m, lmax, ngrid, x, s, DDC_FOLD="1"))
    for et, es in zip(_errors(got, want), _errors(simt, want)):
        assert et <= BAR and et <= 3.0 * es + 1e-7
    if (lmax + 1) ** 2 <= 128:
        assert _differ(got, simt)
    else:
        assert all(np.array_equal(a, b) for a, b in zip(got, simt))
