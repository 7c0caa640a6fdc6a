"""Calls on device vectors whose outputs lie over their inputs: lx and
lstarx together, lx, lstarx, each wholly in place and with a partial overlap, and mkrhs with psi
over the charges, against the same call on vectors of their own.  Bit by bit: only where the
results go differs."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _ptr(t):
    return ctypes.cast(ctypes.c_void_p(t.data_ptr()), ctypes.POINTER(ctypes.c_double))


@pytest.mark.parametrize("prec", [0, 1])
@pytest.mark.parametrize("n,shift", [
    (200, 0), (200, 60),      # lx and lstarx by blocks of their own
    (2500, 0), (2500, 1900),  # by one pass: rows of blocks that start late
    (2500, -1900)])
def test_outputs_over_inputs(n, shift, prec):
    """The output starts `shift` spheres after the input."""
    import torch
    from ddpcm_b200 import molecules as M
    from ddpcm_b200.ddcosmo import DDCosmo
    m = M.to_bohr(M.make_molecule(n, n))
    rng = np.random.default_rng(n)
    nylm = 49
    x, s = (torch.from_numpy(v).cuda() for v in rng.normal(size=(2, n, nylm)))
    with DDCosmo(lmax=6, ngrid=110, eta=0.1, precision=prec, device_pointers=1) as dd:
        pos = [torch.from_numpy(np.ascontiguousarray(m[k])).cuda() for k in "xyzr"]
        torch.cuda.synchronize()
        dd._check(dd.L.ddc_init(dd.h, n, *map(_ptr, pos)))

        def place(v):  # v and an output that lies over it
            buf = torch.zeros(n + abs(shift), nylm, dtype=torch.float64, device="cuda")
            i, o = max(-shift, 0), max(shift, 0)
            buf[i:i + n] = v
            torch.cuda.synchronize()
            return buf[i:i + n], buf[o:o + n]

        y, z = torch.zeros_like(x), torch.zeros_like(s)
        torch.cuda.synchronize()
        dd._check(dd.L.ddc_lx_lstarx(dd.h, _ptr(x), _ptr(y), _ptr(s), _ptr(z)))
        for over_x in (True, False):  # z over x, y over s; y over x, z over s
            x1, ox = place(x)
            s1, os = place(s)
            y1, z1 = (os, ox) if over_x else (ox, os)
            dd._check(dd.L.ddc_lx_lstarx(dd.h, _ptr(x1), _ptr(y1), _ptr(s1), _ptr(z1)))
            assert torch.equal(y1, y) and torch.equal(z1, z)
        for fn, v in ((dd.L.ddc_lx, x), (dd.L.ddc_lstarx, s)):
            want = torch.zeros_like(v)
            torch.cuda.synchronize()
            dd._check(fn(dd.h, _ptr(v), _ptr(want)))
            v1, o1 = place(v)
            dd._check(fn(dd.h, _ptr(v1), _ptr(o1)))
            assert torch.equal(o1, want)


def test_psi_over_the_charges():
    """lmax 0: psi has one entry per charge, and may take the charges' place."""
    import torch
    from ddpcm_b200.ddcosmo import DDCosmo
    rng = np.random.default_rng(5)
    n, nt = 700, 900
    q, x, y, z = (torch.from_numpy(v).cuda() for v in rng.normal(size=(4, n)))
    at = torch.from_numpy(50.0 + rng.normal(size=(nt, 3))).cuda()
    phi, phi1 = torch.zeros(2, nt, dtype=torch.float64, device="cuda")
    psi = torch.zeros_like(q)
    torch.cuda.synchronize()
    with DDCosmo(lmax=0, ngrid=26, device_pointers=1) as dd:
        for f, p in ((phi, psi), (phi1, q)):
            dd._check(dd.L.ddc_mkrhs(dd.h, n, *map(_ptr, (q, x, y, z)), nt, _ptr(at), _ptr(f), 1,
                                     _ptr(p)))
    assert torch.equal(phi1, phi) and torch.equal(q, psi)
