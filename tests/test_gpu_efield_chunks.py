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
