"""Field sums whose source chunks, rounded up to whole tiles, number fewer
than planned: the planned last chunks would start beyond the sources.  FP64
against the oracle's efld (efld.f90:97-114); tolerance 1e-12 relative to the
largest field component (1.5e5 terms, each rounded a few times at 2^-53)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nsrc,ntrg", [(150000, 2560), (150000, 2305), (130817, 2560), (1024, 2560),
                                       (1, 3), (257, 1)])
def test_field_with_rounded_chunks(oracle, nsrc, ntrg):
    from ddpcm_b200.ddcosmo import DDCosmo
    rng = np.random.default_rng(nsrc)
    src = rng.uniform(-0.5, 0.5, nsrc)
    csrc = rng.uniform(-50.0, 50.0, (nsrc, 3))
    ctrg = rng.uniform(55.0, 80.0, (ntrg, 3))
    with DDCosmo(lmax=2, ngrid=26) as dd:
        got = dd.efld(src, csrc, ctrg)
    want = oracle.efld(src, csrc, ctrg)
    assert np.abs(got - want).max() <= 1e-12 * np.abs(want).max()


@pytest.mark.parametrize("nsrc,ntrg", [(587, 12), (64, 1), (65, 1), (1023, 300), (1025, 257),
                                       (16385, 3)])
def test_field_at_few_targets(oracle, nsrc, ntrg):
    """Chunks shorter than a tile (64 sources), up to 16 of them."""
    test_field_with_rounded_chunks(oracle, nsrc, ntrg)


@pytest.mark.parametrize("nsrc,ntrg", [(587, 12), (64, 1), (65, 300), (1025, 257), (30001, 5003),
                                       (150000, 2305)])
def test_potential_in_chunks(oracle, nsrc, ntrg):
    """mkrhs at points of the caller's (mkrhs.f90:102-120), one chunk and
    several; psi goes to the host beside the sum and must come out exactly.
    1e-12 of the largest potential, as above."""
    from ddpcm_b200.ddcosmo import DDCosmo
    rng = np.random.default_rng(nsrc)
    q = rng.uniform(-0.5, 0.5, nsrc)
    src, trg = rng.uniform(-50.0, 50.0, (nsrc, 3)), rng.uniform(55.0, 80.0, (ntrg, 3))
    with DDCosmo(lmax=2, ngrid=26) as dd:
        dd.ddinit(*np.zeros((3, 1)), np.ones(1))
        phi, psi = dd.mkrhs(q, *src.T, ccav=trg)
    want, wpsi = oracle.mkrhs(q, *src.T, trg, 9)
    assert np.abs(phi - want).max() <= 1e-12 * np.abs(want).max()
    np.testing.assert_array_equal(psi, wpsi)


@pytest.mark.parametrize("precision,tol", [(0, 1e-8), (1, 1e-6)])
def test_field_of_a_batch_in_parts(precision, tol):
    """Blocks of 256 nuclei with one, two and three molecules, their sources
    split over parts: forces of the batch against one molecule at a time
    (iconv 10: solutions to 1e-10, taken 100-fold; FP32 pair field 2^-24, taken
    16-fold)."""
    from ddpcm_b200 import molecules as M
    from ddpcm_b200.ddcosmo import DDCosmo
    mols = [M.to_bohr(M.make_molecule(n, 40 + n)) for n in (300, 12, 350)]
    kw = dict(lmax=4, ngrid=50, iconv=10, eta=0.1, precision=precision)
    with DDCosmo(**kw) as dd:
        got = dd.batch_energy_forces(mols)
    with DDCosmo(**kw) as dd:
        for i, m in enumerate(mols):
            one = dd.energy_forces(m["q"], m["x"], m["y"], m["z"], m["r"])
            f = got["fx"][i]
            assert np.linalg.norm(f - one["fx"]) <= tol * np.linalg.norm(one["fx"])
