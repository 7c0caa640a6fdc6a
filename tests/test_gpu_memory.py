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
