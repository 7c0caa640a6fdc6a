"""Routine by routine on a context that a batch has initialised: its spheres
are one system to cosmo (one history, one stop test over all of them, the
report of every iteration), as they are after ddinit."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", [0, 1])
def test_cosmo_after_a_batch(prec):
    from ddpcm_b200 import molecules as M
    from ddpcm_b200.ddcosmo import DDCosmo, PREC_FP64
    mols = [M.to_bohr(M.make_molecule(n, n)) for n in (9, 150)]
    mols[1]["x"] = mols[1]["x"] + 1000.0  # no sphere meets another molecule's
    m = {k: np.concatenate([mol[k] for mol in mols]) for k in "qxyzr"}
    p = dict(lmax=6, ngrid=110, iconv=9, eta=0.1, precision=prec)

    def solve(dd):
        phi, psi = dd.mkrhs(m["q"], m["x"], m["y"], m["z"])
        return [dd.cosmo(star=False, cart=True, phi=phi, psi=psi, return_info=True),
                dd.cosmo(star=True, cart=False, psi=psi, return_info=True)]

    with DDCosmo(**p) as dd:
        dd.ddinit(m["x"], m["y"], m["z"], m["r"])
        want = solve(dd)
    with DDCosmo(**p) as dd:
        dd.batch_energy_forces(mols)
        a = [ctypes.c_int() for _ in range(4)]
        dd._check(dd.L.ddc_sizes(dd.h, *map(ctypes.byref, a)))
        dd.nsph, dd.ncav, dd.nylm, dd.ngrid = (v.value for v in a)
        got = solve(dd)
    for (x, e, i), (xw, ew, iw) in zip(got, want):
        assert np.array_equal(x, xw) and e == ew
        for k in ("iterations", "converged", "refinements", "final_norm"):
            assert i[k] == iw[k]
        assert list(i["norms"]) == list(iw["norms"]) and len(i["norms"]) == i["iterations"]
        if prec == PREC_FP64:
            assert i["norms"][-1] == i["final_norm"] < 1e-9
