"""Device memory that a call takes beyond its arguments."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _ptr(t):
    return ctypes.cast(ctypes.c_void_p(t.data_ptr()), ctypes.POINTER(ctypes.c_double))


def test_potential_at_many_points():
    """Many targets on device arrays: the sources are taken in one piece, which
    needs no partial sums (8 bytes per target otherwise: 320 MB)."""
    import torch
    from ddpcm_b200.ddcosmo import DDCosmo
    nt = 40_000_000
    q, x, y, z = torch.zeros(4, 1, dtype=torch.float64, device="cuda")
    q.fill_(2.0)
    psi = torch.zeros_like(q)
    at = torch.ones(nt, 3, dtype=torch.float64, device="cuda")
    phi = torch.zeros(nt, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    with DDCosmo(lmax=0, ngrid=26, device_pointers=1) as dd:
        def call(n):
            dd._check(dd.L.ddc_mkrhs(dd.h, 1, *map(_ptr, (q, x, y, z)), n, _ptr(at), _ptr(phi), 1,
                                     _ptr(psi)))
        call(1)  # kernels loaded
        free = torch.cuda.mem_get_info()[0]
        call(nt)
        assert free - torch.cuda.mem_get_info()[0] < 50e6
    assert abs(float(phi[-1]) - 2.0 / np.sqrt(3.0)) < 1e-15
    assert bool((phi == phi[-1]).all())


@pytest.mark.parametrize("iprint", [0, 1])
@pytest.mark.parametrize("prec", [0, 1])
def test_iteration_budget_costs_no_memory(prec, iprint):
    """A budget that is not meant to run out: the log of increment norms is
    bounded (8 bytes per allowed iteration and system otherwise: 32 GB)."""
    import torch
    from ddpcm_b200 import molecules as M
    from ddpcm_b200.ddcosmo import DDCosmo
    m = M.to_bohr(M.make_molecule(12, 4))
    p = dict(lmax=6, ngrid=110, iconv=8, eta=0.1, precision=prec, iprint=iprint)

    def solve(dd):
        out = dd.energy_forces(*(m[k] for k in "qxyzr"))
        return out, torch.cuda.mem_get_info()[0]

    with DDCosmo(**p) as dd:
        want, free = solve(dd)
    with DDCosmo(max_iter=2_000_000_000, **p) as dd:
        got, free1 = solve(dd)
    assert free - free1 < 200e6
    assert np.array_equal(got["sigma"], want["sigma"]) and np.array_equal(got["s"], want["s"])
    for side in ("direct", "adjoint"):
        a, b = got["info"][side], want["info"][side]
        assert list(a["norms"]) == list(b["norms"]) and len(a["norms"]) == a["iterations"]


@pytest.mark.parametrize("prec", [0, 1])
def test_iterations_beyond_the_report(prec):
    """More iterations than a report holds: the first 256 norms, as ever."""
    from ddpcm_b200 import molecules as M
    from ddpcm_b200.ddcosmo import DDCosmo
    m = M.to_bohr(M.make_molecule(60, 100))
    p = dict(lmax=6, ngrid=110, iconv=10, eta=0.1, precision=prec, ndiis=0)
    with DDCosmo(max_iter=5000, **p) as dd:
        out = dd.energy_forces(*(m[k] for k in "qxyzr"))
    i = out["info"]["direct"]
    assert i["converged"]
    norms = list(i["norms"])
    assert len(norms) == min(i["iterations"], 256) and all(v > 0.0 for v in norms)
