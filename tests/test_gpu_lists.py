"""The list building of ddinit at the edges of its one-block scan (8,192
counts per step, 32,768 counts in all): chains of n spheres have 2 (n - 1)
neighbour pairs.  Cavity points and operators against the oracle
(ddcosmo.f90:159-483, matvec.f90:94-235), on one context from size to size,
so that the tables kept with the context serve every molecule.

Tolerances: points 1e-12, four roundings at coordinates up to 1,300; operators
1e-13 relative in the 2-norm as elsewhere."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes", [(4097, 1, 4098, 2), (16385, 16386), (32768, 32769)])
def test_chains_at_the_edges_of_the_scan(oracle, sizes):
    from ddpcm_b200.ddcosmo import DDCosmo
    lmax, ngrid = 2, 26
    with DDCosmo(lmax=lmax, ngrid=ngrid, iconv=10, eta=0.1) as dd:
        for n in sizes:
            x = 2.0 * (np.arange(n) % 128)           # rows of 128 along x, stacked in y
            y = 5.0 * (np.arange(n) // 128)
            z, r = np.zeros(n), np.full(n, 1.5)
            ref = oracle.RefDD(lmax, ngrid, 10, 1, 78.3553, 0.1).init(x, y, z, r)
            dd.ddinit(x, y, z, r)
            assert dd.ncav == ref.ncav
            assert np.max(np.abs(dd.ccav - ref.get("ccav"))) <= 1e-12
            v, s = np.random.default_rng(n).normal(size=(2, n, (lmax + 1) ** 2))
            for got, want in zip(dd.lx_lstarx(v, s), (ref.lx(v), ref.lstarx(s))):
                assert np.linalg.norm(got - want) <= 1e-13 * np.linalg.norm(want)


@pytest.mark.parametrize("sizes", [(1184, 1185), (65537,)])
def test_where_the_passes_take_the_longest_lists_first(oracle, sizes):
    """Spheres in order, sorted (1,185 to 65,536, the sizes above) and in order
    again: every sphere's list must be taken once."""
    test_chains_at_the_edges_of_the_scan(oracle, sizes)
