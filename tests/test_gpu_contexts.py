"""Contexts of different parameters that live side by side in one process:
what one of them sets for the device's kernels must leave the others as they
were.  A context's results after another one has been initialised and used
are the results it gave alone, bit by bit (sums have a fixed order)."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _molecule(n, seed):
    from ddpcm_b200 import molecules as M
    return M.to_bohr(M.make_molecule(n, seed))


def _results(dd, m):
    out = dd.energy_forces(*(m[k] for k in "qxyzr"))
    phi, psi = dd.mkrhs(m["q"], m["x"], m["y"], m["z"])
    pair = dd.lx_lstarx(out["sigma"], out["s"])
    return [np.float64(out["esolv"]), out["sigma"], out["s"], out["fx"], dd.rhs(phi), psi, *pair,
            dd.ddmkzeta(out["s"])]


def _same(a, b):
    assert all(np.array_equal(u, v) for u, v in zip(a, b))


@pytest.mark.parametrize("prec", [0, 1])
@pytest.mark.parametrize("wide,narrow", [((10, 590), (6, 110)), ((12, 1202), (2, 50)),
                                         ((9, 434), (10, 302))])
def test_two_live_contexts(wide, narrow, prec):
    """More grid points (more shared memory in the folded contractions) in the
    first context, fewer in the second."""
    from ddpcm_b200.ddcosmo import DDCosmo
    m = _molecule(40, 1)
    with DDCosmo(lmax=wide[0], ngrid=wide[1], eta=0.1, precision=prec) as a:
        first = _results(a, m)
        with DDCosmo(lmax=narrow[0], ngrid=narrow[1], eta=0.1, precision=prec) as b:
            other = _results(b, m)
            _same(_results(a, m), first)
            _same(_results(b, m), other)
        _same(_results(a, m), first)


def test_two_live_contexts_on_tcgen05():
    """Mixed operators above 2e8 products, where the contractions run on
    tcgen05: wide tiles (14,000 spheres), then narrow ones (2,900)."""
    from ddpcm_b200.ddcosmo import DDCosmo, PREC_MIXED

    def pair(dd, n, lmax):
        rng = np.random.default_rng(n)
        return dd.lx_lstarx(*rng.normal(size=(2, n, (lmax + 1) ** 2)))

    def context(n, lmax, ngrid):
        m = _molecule(n, n)
        return DDCosmo(lmax=lmax, ngrid=ngrid, eta=0.1, precision=PREC_MIXED).ddinit(
            m["x"], m["y"], m["z"], m["r"])

    with context(14000, 6, 302) as a:
        first = pair(a, 14000, 6)
        with context(2900, 10, 590) as b:
            other = pair(b, 2900, 10)
            _same(pair(a, 14000, 6), first)
            _same(pair(b, 2900, 10), other)


def test_contexts_of_several_threads():
    """Four threads, each with a context of its own on a grid whose point lists
    take more than the default 48 KB of shared memory."""
    from ddpcm_b200.ddcosmo import DDCosmo
    m = _molecule(4, 3)
    failed = []

    def work(ngrid):
        try:
            with DDCosmo(lmax=2, ngrid=ngrid, eta=0.1) as dd:
                for _ in range(2000):
                    dd.ddinit(m["x"], m["y"], m["z"], m["r"])
        except Exception as e:  # reported by the main thread
            failed.append(f"{ngrid}: {e}")

    threads = [threading.Thread(target=work, args=(g,)) for g in (3074, 5810, 3470, 5294)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed, failed
