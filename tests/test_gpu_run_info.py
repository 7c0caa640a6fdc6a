"""What a run reports without waiting for each phase: phase times that are
positive and add up to no more than the call, and results that do not depend
on the solves running side by side or on where the output arrays lie.  The two
orders of solving share every kernel's arithmetic except the fused pass;
iconv 10 leaves 1e-10, taken 100-fold."""
import ctypes
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("igrad", [0, 1])
@pytest.mark.parametrize("precision", [0, 1])
def test_phases_and_results(precision, igrad):
    from ddpcm_b200 import molecules as M
    from ddpcm_b200.ddcosmo import DDCosmo
    m = M.to_bohr(M.make_molecule(60, 77))
    args = [m[k] for k in ("q", "x", "y", "z", "r")]
    got = []
    for pair in (1, 0):
        with DDCosmo(lmax=6, ngrid=110, iconv=10, eta=0.1, igrad=igrad, precision=precision,
                     pair_solves=pair) as dd:
            for _ in range(3):
                t = time.perf_counter()
                r = dd.energy_forces(*args)
                t = time.perf_counter() - t
                i = r["info"]
                parts = [i[k] for k in ("t_init", "t_mkrhs", "t_direct", "t_adjoint", "t_forces")]
                assert min(parts[:3]) > 0 and min(parts) >= 0
                assert sum(parts) <= t
            got.append(r)
    a, b = got
    assert abs(a["esolv"] - b["esolv"]) <= 1e-8 * abs(b["esolv"])
    for k in ("sigma", "s", "fx"):
        assert np.linalg.norm(a[k] - b[k]) <= (1e-8 if precision == 0 else 1e-7) \
            * np.linalg.norm(b[k])


def test_no_convergence_still_reports_its_times():
    from ddpcm_b200 import molecules as M
    from ddpcm_b200.ddcosmo import DDCosmo, RunInfo, _p as p
    m = M.to_bohr(M.make_molecule(20, 78))
    with DDCosmo(lmax=4, ngrid=50, iconv=12, eta=0.1, max_iter=2) as dd:
        q, x, y, z, r = (np.ascontiguousarray(m[k], dtype=np.float64) for k in
                         ("q", "x", "y", "z", "r"))
        sig, s = np.full((2, 20, 25), 7.0)
        fx, e, info = np.zeros((20, 3)), ctypes.c_double(3.0), RunInfo()
        st = dd.L.ddc_energy_forces(dd.h, 20, p(q), p(x), p(y), p(z), p(r), ctypes.byref(e),
                                    p(sig), p(s), p(fx), ctypes.byref(info))
        assert st != 0 and info.t_init > 0 and info.t_mkrhs > 0
        assert e.value == 3.0 and np.all(sig == 7.0) and np.all(s == 7.0)
