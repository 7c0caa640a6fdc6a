"""Workloads of the ddCOSMO library for performance measurement.

Each case is what a program that uses the library has it do, through the
public entry points of ``ddpcm_b200``:

* ``flow``: energy and forces of one molecule in one call
  (``ddc_energy_forces``: ddinit, right-hand side, direct and adjoint solve,
  forces), on host arrays or on device arrays;
* ``staged``: the same through the separate routines that the reference's
  main program calls one after the other;
* ``batch``: many independent molecules in one ``ddc_batch_energy_forces``;
* ``operators``: one application of L and / or L* to device vectors, as in a
  program with an iterative solver of its own;
* ``charges``: potential and field of point charges at the points of another
  set (``mkrhs`` and ``efld`` with the program's own coordinates).

Molecules are the package's seeded globules (0.1 atoms per cubic angstrom) and
chains; eta and eps are the benchmark's.  The solves stop at an increment of
10^-12, as a program asks for that differentiates the forces once more or
follows energy conservation over a long trajectory.
"""
import ctypes
import math
import os
import re

import numpy as np
import torch

from ddpcm_b200 import ddcosmo, molecules
from ddpcm_b200.ddcosmo import DDCosmo

ETA, EPS, ICONV = 0.1, 78.3553, 12
GRIDS = (110, 146, 170, 194, 230, 266, 302, 350, 434, 590)


def listed():
    return [
        # the smallest call: a dozen atoms, where a host program waits for
        # launches and round trips (a scan over conformers, a unit test)
        dict(name="chain12_fp64", kind="flow", n=12, globule=False, lmax=6, ngrid=110,
             precision="fp64", start="reference", device=False),
        # a drug-sized molecule in mixed precision
        dict(name="drug113_mixed", kind="flow", n=113, globule=True, lmax=6, ngrid=110,
             precision="mixed", start="reference", device=False),
        # a small protein at the accuracy of the mixed-precision benchmark
        dict(name="protein600_mixed", kind="flow", n=600, globule=True, lmax=8, ngrid=302,
             precision="mixed", start="reference", device=False),
        # a host program that replaces the Fortran module routine by routine
        dict(name="staged643_fp64", kind="staged", n=643, lmax=6, ngrid=110),
        # a medium protein, all in FP64
        dict(name="protein2000_fp64", kind="flow", n=2000, globule=True, lmax=6, ngrid=302,
             precision="fp64", start="reference", device=False),
        # one frame of molecular dynamics from the previous frame's solutions;
        # an odd degree and an odd number of atoms
        dict(name="frame1999_mixed", kind="flow", n=1999, globule=True, lmax=7, ngrid=194,
             precision="mixed", start="previous", device=False),
        # a large protein in FP64
        dict(name="globule5000_fp64", kind="flow", n=5000, globule=True, lmax=10, ngrid=590,
             precision="fp64", start="reference", device=False),
        # the benchmark's large single solve, inputs and outputs on the device
        dict(name="globule20000_mixed", kind="flow", n=20000, globule=True, lmax=10, ngrid=590,
             precision="mixed", start="reference", device=True),
        # a screening batch of small molecules in FP64
        dict(name="batch64_fp64", kind="batch", count=64, lo=20, hi=200, lmax=6, ngrid=110,
             precision="fp64"),
        # a batch of very uneven sizes in mixed precision
        dict(name="batch48_mixed", kind="batch", count=48, lo=20, hi=2000, lmax=6, ngrid=302,
             precision="mixed"),
        # one paired operator application of an external solver
        dict(name="operators4999_fp64", kind="operators", n=4999, lmax=9, ngrid=434, op="pair"),
        # QM/MM electrostatics: a solvent's charges at a cavity's points
        dict(name="charges_fp64", kind="charges", nsrc=30001, ntrg=50003),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("flow", "flow", "flow", "flow", "staged", "batch", "batch", "operators",
                       "charges"))
    if kind == "charges":
        return dict(kind=kind, nsrc=_log(rng, 500, 60000), ntrg=_log(rng, 500, 60000))
    # degree and grid go together: the grid integrates the products of the
    # harmonics it has to resolve
    lmax = rng.randint(6, 10)
    ngrid = rng.choice([g for g in GRIDS if g >= 1.4 * (lmax + 1) ** 2])
    if kind == "flow":
        n = _log(rng, 8, 6000)
        return dict(kind=kind, n=n, globule=n > 30 or rng.random() < 0.5, lmax=lmax, ngrid=ngrid,
                    precision=rng.choice(("fp64", "mixed")),
                    start=rng.choice(("reference", "reference", "previous")),
                    device=rng.random() < 0.3)
    if kind == "staged":
        return dict(kind=kind, n=_log(rng, 8, 3000), lmax=lmax, ngrid=ngrid)
    if kind == "batch":
        hi = _log(rng, 60, 2000)
        return dict(kind=kind, count=_log(rng, 4, 64), lo=max(5, hi // rng.randint(2, 60)), hi=hi,
                    lmax=rng.randint(6, 7), ngrid=rng.choice((110, 194, 302)),
                    precision=rng.choice(("fp64", "mixed")))
    return dict(kind=kind, n=_log(rng, 200, 8000), lmax=lmax, ngrid=ngrid,
                op=rng.choice(("pair", "pair", "lx", "lstarx")))


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _molecule(case, seed):
    return molecules.make_molecule(case["n"], seed, globule=case.get("globule", True))


def _frames(case, seed):
    """The molecules of a case that starts from a previous frame, in bohr:
    that frame, then the one to solve."""
    mol = _molecule(case, seed)
    return [molecules.to_bohr(f) for f in molecules.trajectory(mol, 2, seed=seed + 1)]


def _solved(case, seed):
    if case.get("start") == "previous":
        return _frames(case, seed)[1]
    return molecules.to_bohr(_molecule(case, seed))


def _batch(case, seed):
    """Globules of log-uniform sizes (the same sizes for every seed)."""
    rng = np.random.default_rng(case["count"])
    sizes = np.exp(rng.uniform(math.log(case["lo"]), math.log(case["hi"]), case["count"])).astype(int)
    return [molecules.to_bohr(molecules.make_molecule(int(n), 1000 * seed + k))
            for k, n in enumerate(sizes)]


def _vectors(case, seed):
    """Two vectors of the size and decay of solutions: order 0.1 per sphere,
    smaller with the degree."""
    rng = np.random.default_rng(seed + 7)
    scale = np.concatenate([np.full(2 * l + 1, 0.1 / (1 + l) ** 2) for l in range(case["lmax"] + 1)])
    return [scale * rng.normal(size=(case["n"], len(scale))) for _ in range(2)]


def _charges(case, seed):
    """Charges in a box at the density of water's sites, targets outside a
    closest approach of 2 bohr to any lattice site."""
    rng = np.random.default_rng(seed)
    side = math.ceil(case["nsrc"] ** (1 / 3))
    site = np.stack(np.meshgrid(*[np.arange(side)] * 3, indexing="ij"), -1).reshape(-1, 3)
    a = 4.0  # bohr between lattice sites
    src = a * site[rng.permutation(len(site))[: case["nsrc"]]] + rng.uniform(-0.4, 0.4, (case["nsrc"], 3))
    cell = rng.integers(0, side, (case["ntrg"], 3))
    trg = a * (cell + 0.5) + rng.uniform(-0.4, 0.4, (case["ntrg"], 3))
    q = rng.uniform(-0.5, 0.5, case["nsrc"])
    return q - q.mean(), src, trg


def _context(case, **more):
    prec = ddcosmo.PREC_MIXED if case.get("precision") == "mixed" else ddcosmo.PREC_FP64
    return DDCosmo(lmax=case["lmax"], ngrid=case["ngrid"], iconv=ICONV, eta=ETA, eps=EPS,
                   precision=prec, **more)


def _device(a):
    return torch.from_numpy(np.array(a, dtype=np.float64)).cuda()


def prepare(case, seed):
    kind = case["kind"]
    if kind == "flow":
        previous = case["start"] == "previous"
        mol = _solved(case, seed)
        state = dict(case=case, mol=mol)
        if previous:
            first = _frames(case, seed)[0]
            with _context(case) as dd:
                out = dd.energy_forces(*(first[k] for k in "qxyzr"))
            state["sigma"], state["s"] = out["sigma"], out["s"]
        state["dd"] = _context(case, device_pointers=int(case["device"]),
                               guess=ddcosmo.GUESS_USER if previous else ddcosmo.GUESS_REFERENCE)
        if case["device"]:
            nylm = (case["lmax"] + 1) ** 2
            state["in"] = [_device(mol[k]) for k in "qxyzr"]
            state["out"] = [torch.zeros(case["n"], w, dtype=torch.float64, device="cuda")
                            for w in (nylm, nylm, 3)]
            if previous:
                state["guess"] = [_device(state[k]) for k in ("sigma", "s")]
        return state
    if kind == "staged":
        return dict(case=case, mol=_solved(case, seed), dd=_context(case))
    if kind == "batch":
        return dict(case=case, mols=_batch(case, seed), dd=_context(case))
    if kind == "operators":
        mol = _solved(case, seed)
        dd = _context(case, device_pointers=1)
        pos = [_device(mol[k]) for k in "xyzr"]
        dd._check(dd.L.ddc_init(dd.h, case["n"], *map(_ptr, pos)))
        x, s = (_device(v) for v in _vectors(case, seed))
        return dict(case=case, dd=dd, x=x, s=s, y=torch.zeros_like(x), z=torch.zeros_like(s))
    # the context of the solute that the charges surround
    q, src, trg = _charges(case, seed)
    mol = molecules.to_bohr(molecules.make_molecule(24, seed))
    dd = DDCosmo(lmax=6, ngrid=110).ddinit(mol["x"], mol["y"], mol["z"], mol["r"])
    return dict(case=case, q=q, src=src, trg=trg, dd=dd)


def _ptr(t):
    return ctypes.cast(ctypes.c_void_p(t.data_ptr()), ctypes.POINTER(ctypes.c_double))


def run(state):
    case, dd = state["case"], state["dd"]
    kind = case["kind"]
    if kind == "flow":
        if case["device"]:
            sigma, s, fx = state["out"]
            if "guess" in state:  # the outputs carry the start in
                sigma.copy_(state["guess"][0])
                s.copy_(state["guess"][1])
                torch.cuda.current_stream().synchronize()
            r = dd.energy_forces_ptr(*(t.data_ptr() for t in state["in"]), case["n"],
                                     sigma.data_ptr(), s.data_ptr(), fx.data_ptr())
            return dict(esolv=np.float64(r["esolv"]), sigma=sigma, s=s, fx=fx)
        r = dd.energy_forces(*(state["mol"][k] for k in "qxyzr"), sigma0=state.get("sigma"),
                             s0=state.get("s"))
        return dict(esolv=np.float64(r["esolv"]), sigma=r["sigma"], s=r["s"], fx=r["fx"])
    if kind == "staged":  # main.f90:164-265
        m = state["mol"]
        dd.ddinit(m["x"], m["y"], m["z"], m["r"])
        phi, psi = dd.mkrhs(m["q"], m["x"], m["y"], m["z"])
        sigma, esolv = dd.cosmo(star=False, cart=True, phi=phi, psi=psi)
        s, _ = dd.cosmo(star=True, cart=False, psi=psi)
        fx = dd.forces_dd(phi, sigma, s)
        zeta = dd.ddmkzeta(s)
        centres, cavity = dd.csph, dd.ccav
        e_solute = dd.efld(m["q"], centres, cavity)
        e_zeta = dd.efld(zeta, cavity, centres)
        owner = np.nonzero(dd.ui > 0.0)[0]
        for k in range(3):
            fx[:, k] -= np.bincount(owner, zeta * e_solute[:, k], case["n"]) + m["q"] * e_zeta[:, k]
        return dict(esolv=np.float64(esolv), sigma=sigma, s=s, e_zeta=e_zeta, fx=fx)
    if kind == "batch":
        r = dd.batch_energy_forces(state["mols"])
        return dict(esolv=r["esolv"], fx=np.concatenate(r["fx"]))
    if kind == "operators":
        x, s, y, z = state["x"], state["s"], state["y"], state["z"]
        if case["op"] == "pair":
            dd._check(dd.L.ddc_lx_lstarx(dd.h, _ptr(x), _ptr(y), _ptr(s), _ptr(z)))
            return dict(y=y, z=z)
        if case["op"] == "lx":
            dd._check(dd.L.ddc_lx(dd.h, _ptr(x), _ptr(y)))
            return dict(y=y)
        dd._check(dd.L.ddc_lstarx(dd.h, _ptr(s), _ptr(z)))
        return dict(z=z)
    phi, _ = dd.mkrhs(state["q"], *state["src"].T, ccav=state["trg"])
    return dict(phi=phi, ef=dd.efld(state["q"], state["src"], state["trg"]))


# ---------------------------------------------------------------------------
# the work of one pass
# ---------------------------------------------------------------------------
def _flow_work(n, lmax, ngrid, solves=2, iterations=45):
    """A globule has about 3 (point, containing neighbour) pairs per grid
    point and 0.15 cavity points per grid point; each iteration evaluates
    every harmonic at every such pair (3 operations) and contracts it with
    the two systems' vectors (2 multiply-adds each), projects and expands."""
    y = (lmax + 1) ** 2
    triples = 3.0 * n * ngrid
    ncav = 0.15 * n * ngrid
    per_it = triples * y * (1.5 + 2.0 * solves) + 2.0 * y * ngrid * n * solves
    vectors = 8.0 * n * y * (2 + solves)
    return dict(bytes=8.0 * 8 * n + vectors + 24.0 * n,
                flops=iterations * per_it + ncav * min(n, 3000) * 38.0)


def work(case):
    kind = case["kind"]
    if kind == "charges":
        ns, nt = case["nsrc"], case["ntrg"]
        return dict(bytes=8.0 * (4 * ns * 2 + 3 * nt * 2 + 4 * nt), flops=32.0 * ns * nt)
    if kind == "batch":
        lo, hi = case["lo"], case["hi"]
        mean = (hi - lo) / math.log(hi / lo)
        return _flow_work(case["count"] * mean, case["lmax"], case["ngrid"], iterations=40)
    if kind == "operators":
        n, y, g = case["n"], (case["lmax"] + 1) ** 2, case["ngrid"]
        both = 2 if case["op"] == "pair" else 1
        return dict(bytes=16.0 * n * y * both,
                    flops=3.0 * n * g * y * (1.5 + 2.0 * both) + 2.0 * y * g * n * both)
    its = 25 if case.get("start") == "previous" else 20 + 4.5 * math.log2(max(case["n"], 8))
    return _flow_work(case["n"], case["lmax"], case["ngrid"], iterations=its)


# ---------------------------------------------------------------------------
# exact values: the ddCOSMO equations in 64 bits with plain torch.  The
# forces are the derivative of the discrete energy by automatic
# differentiation of S.(g - L X).
# ---------------------------------------------------------------------------
def _lebedev(ngrid):
    """Points and 4 pi weights of the Lebedev-Laikov rule, from the published
    orbit parameters and in the order in which the cavity is indexed."""
    path = os.path.join(os.path.dirname(ddcosmo.__file__), "csrc", "lebedev_orbits.inc")
    text = open(path).read()
    ints = {k: [int(v) for v in re.search(k + r"\[\w+\] = \{([^}]*)\}", text).group(1).split(",")]
            for k in ("leb_sizes", "leb_orbit_off", "leb_orbit_cnt")}
    recs = re.findall(r"\{(\d), ([^,]+), ([^,]+), ([^}]+)\}", text[text.index("leb_orbits["):])
    at = ints["leb_sizes"].index(ngrid)
    first, count = ints["leb_orbit_off"][at], ints["leb_orbit_cnt"][at]
    shapes = {1: ("a00", "0a0", "00a"), 2: ("0aa", "a0a", "aa0"), 3: ("aaa",),
              4: ("aab", "aba", "baa"), 5: ("ab0", "ba0", "a0b", "b0a", "0ab", "0ba"),
              6: ("abc", "acb", "bac", "bca", "cab", "cba")}
    pts = []
    for code, a, b, v in recs[first:first + count]:
        code, a, b, v = int(code), float(a), float(b), float(v)
        if code <= 3:
            a = math.sqrt(1.0 / code)
        elif code == 4:
            b = math.sqrt(1.0 - 2.0 * a * a)
        elif code == 5:
            b = math.sqrt(1.0 - a * a)
        value = {"0": 0.0, "a": a, "b": b, "c": math.sqrt(max(0.0, 1.0 - a * a - b * b))}
        for shape in shapes[code]:
            nz = [k for k in range(3) if shape[k] != "0"]
            for sign in range(1 << len(nz)):
                p = [value[c] for c in shape]
                for i, k in enumerate(nz):
                    if sign >> i & 1:
                        p[k] = -p[k]
                pts.append(p + [4.0 * math.pi * v])
    assert len(pts) == ngrid
    return np.array(pts)


def _harmonics(p, lmax):
    """Real solid harmonics r^l Y_lm of the points p[q, 3], columns l*l+l+m."""
    x, y, z = p.unbind(1)
    r2 = x * x + y * y + z * z
    col = [None] * (lmax + 1) ** 2
    re, im = torch.ones_like(x), torch.zeros_like(x)
    for m in range(lmax + 1):
        if m:
            re, im = re * x - im * y, re * y + im * x
        p0, p1 = torch.zeros_like(x), torch.full_like(x, math.prod(range(1, 2 * m, 2)))
        for l in range(m, lmax + 1):
            if l > m:
                p0, p1 = p1, ((2 * l - 1) * z * p1 - (l + m - 1) * r2 * p0) / (l - m)
            c = math.sqrt((2 * l + 1) / (4 * math.pi) * math.factorial(l - m) / math.factorial(l + m))
            if m:
                c *= math.sqrt(2.0)
                col[l * l + l - m] = c * im * p1
            col[l * l + l + m] = c * re * p1
    return torch.stack(col, 1)


def _switch(t):
    a, b = 15.0 * ETA - 12.0, 10.0 * ETA * ETA - 15.0 * ETA + 6.0
    mid = (1.0 - t) ** 3 * (6.0 * t * t + a * t + b) / ETA ** 5
    return torch.where(t <= 1.0 - ETA, torch.ones_like(t), torch.where(t < 1.0, mid, torch.zeros_like(t)))


class _Exact:
    """The discretised problem of one or more molecules."""
    MOST = 1.2e9  # harmonics held

    def __init__(self, mols, lmax, ngrid):
        self.dev = "cuda" if torch.cuda.is_available() else "cpu"
        put = lambda a: torch.as_tensor(np.asarray(a, dtype=np.float64), device=self.dev)  # noqa: E731
        cat = {k: put(np.concatenate([m[k] for m in mols])) for k in "qxyzr"}
        self.c = torch.stack([cat[k] for k in "xyz"], 1)
        self.r, self.q = cat["r"], cat["q"]
        self.mol = torch.repeat_interleave(torch.arange(len(mols), device=self.dev),
                                           torch.tensor([len(m["q"]) for m in mols], device=self.dev))
        self.n, self.lmax, self.nmol = len(self.r), lmax, len(mols)
        grid = put(_lebedev(ngrid))
        self.s, self.w, self.g = grid[:, :3], grid[:, 3], ngrid
        self.basis = _harmonics(self.s, lmax)
        self.facl = put(np.concatenate([np.full(2 * l + 1, (2 * l + 1) / (4 * math.pi))
                                        for l in range(lmax + 1)]))
        d = torch.cdist(self.c, self.c)
        near = (d < self.r[:, None] + self.r[None]) & (self.mol[:, None] == self.mol[None])
        near.fill_diagonal_(False)
        pairs = near.nonzero()
        parts = []
        for k in range(0, len(pairs), 20000):
            a, b = pairs[k:k + 20000].unbind(1)
            v = (self.c[a] - self.c[b])[:, None] + self.r[a][:, None, None] * self.s[None]
            hit = (v.norm(dim=2) < self.r[b][:, None]).nonzero()
            parts.append(torch.stack([a[hit[:, 0]], hit[:, 1], b[hit[:, 0]]], 1))
        # the triples, sphere by sphere
        self.a, self.p, self.b = (torch.cat(parts) if parts else pairs.new_zeros((0, 3))).unbind(1)
        self.row = self.a * ngrid + self.p
        self.f, W = self._weights(self.c, slice(None))
        self.u = torch.where(self.f <= 1.0, 1.0 - self.f, torch.zeros_like(self.f))
        self.size = len(self.a) * self.basis.shape[1]
        if self.size > self.MOST:
            return
        self.step = 400000
        self.Y = torch.empty(len(self.a), self.basis.shape[1], dtype=torch.float64, device=self.dev)
        for k in range(0, len(self.a), self.step):
            q = slice(k, k + self.step)
            self.Y[q] = W[q, None] * _harmonics(self._scaled(self.c, q), lmax) / self.facl

    def _scaled(self, c, q):
        a, b = self.a[q], self.b[q]
        return (c[a] - c[b] + self.r[a, None] * self.s[self.p[q]]) / self.r[b, None]

    def _weights(self, c, q):
        chi = _switch(self._scaled(c, q).norm(dim=1))
        f = torch.zeros(self.n * self.g, dtype=torch.float64, device=self.dev)
        f = f.index_add(0, self.row[q], chi)
        at = f[self.row[q]]
        return f, torch.where(at > 1.0, chi / at, chi)

    def lx(self, x):
        """Off-diagonal L x."""
        v = torch.zeros(self.n * self.g, dtype=torch.float64, device=self.dev)
        for k in range(0, len(self.a), self.step):
            q = slice(k, k + self.step)
            v.index_add_(0, self.row[q], (self.Y[q] * x[self.b[q]]).sum(1))
        return -(v.view(self.n, self.g) * self.w) @ self.basis

    def lstarx(self, s):
        """Off-diagonal L* s."""
        xi = (s @ self.basis.T * self.w).reshape(-1)
        y = torch.zeros_like(s)
        for k in range(0, len(self.a), self.step):
            q = slice(k, k + self.step)
            y.index_add_(0, self.b[q], self.Y[q] * xi[self.row[q], None])
        return -y

    def solve(self, op, rhs):
        """(1/facl + op) x = rhs by restarted GMRES on the equation scaled by
        facl, to the rounding of the residual."""
        b = self.facl * rhs
        x = torch.zeros_like(b)
        for _ in range(4):
            r = b - x - self.facl * op(x)
            beta = r.norm()
            if not len(b) or beta <= 1e-15 * b.norm():
                break
            m = 90
            V = torch.zeros(m + 1, b.numel(), dtype=torch.float64, device=self.dev)
            H = np.zeros((m + 1, m))
            V[0] = (r / beta).reshape(-1)
            for j in range(m):
                v = V[j].view_as(b)
                t = (v + self.facl * op(v)).reshape(-1)
                for _ in range(2):
                    h = V[:j + 1] @ t
                    t = t - V[:j + 1].T @ h
                    H[:j + 1, j] += h.cpu().numpy()
                H[j + 1, j] = float(t.norm())
                e = np.zeros(j + 2)
                e[0] = float(beta)
                k, res = np.linalg.lstsq(H[:j + 2, :j + 1], e, rcond=None)[:2]
                left = np.linalg.norm(H[:j + 2, :j + 1] @ k - e)
                if left < 1e-15 * float(b.norm()) or H[j + 1, j] < 1e-14:
                    break
                V[j + 1] = t / H[j + 1, j]
            x = x + (torch.as_tensor(k, device=self.dev) @ V[:len(k)]).view_as(b)
        return x

    def cavity(self):
        """Indices of the cavity points (sphere, point) and their positions."""
        at = (self.u > 0.0).nonzero()[:, 0]
        a, p = at // self.g, at % self.g
        return at, a, self.c[a] + self.r[a, None] * self.s[p]

    def potential(self):
        at, a, pos = self.cavity()
        phi = torch.zeros(len(at), dtype=torch.float64, device=self.dev)
        for k in range(self.nmol):
            t, j = (self.mol[a] == k).nonzero()[:, 0], (self.mol == k).nonzero()[:, 0]
            phi[t] = _coulomb(self.q[j], self.c[j], pos[t])[0]
        return phi

    def fields(self, zeta):
        """Field of the charges at the cavity and of zeta at the nuclei."""
        _, a, pos = self.cavity()
        e, z = torch.zeros_like(pos), torch.zeros_like(self.c)
        for k in range(self.nmol):
            t, j = (self.mol[a] == k).nonzero()[:, 0], (self.mol == k).nonzero()[:, 0]
            e[t] = _coulomb(self.q[j], self.c[j], pos[t])[1]
            z[j] = _coulomb(zeta[t], pos[t], self.c[j])[1]
        return e, z

    def solution(self):
        """X, S and the energies of the molecules."""
        phi = self.potential()
        grid = torch.zeros(self.n * self.g, dtype=torch.float64, device=self.dev)
        grid[self.cavity()[0]] = phi
        self.phi_grid = grid
        rhs = -((self.u * grid).view(self.n, self.g) * self.w) @ self.basis
        psi = torch.zeros_like(rhs)
        psi[:, 0] = math.sqrt(4.0 * math.pi) * self.q
        x, s = self.solve(self.lx, rhs), self.solve(self.lstarx, psi)
        fep = 0.5 * (EPS - 1.0) / EPS
        e = torch.zeros(self.nmol, dtype=torch.float64, device=self.dev)
        e.index_add_(0, self.mol, fep * (x * psi).sum(1))
        return x, s, e

    def forces(self, x, s):
        """Forces, and the field of zeta at the nuclei."""
        fep = 0.5 * (EPS - 1.0) / EPS
        wxi = (s @ self.basis.T * self.w).reshape(-1)
        grad = torch.zeros_like(self.c)
        ends = torch.searchsorted(self.a.contiguous(), torch.arange(self.n + 1, device=self.dev)).tolist()
        lo = 0
        while lo < self.n:
            hi = lo + 1
            while hi < self.n and ends[hi + 1] - ends[lo] <= 150000:
                hi += 1
            q = slice(ends[lo], ends[hi])
            if ends[hi] > ends[lo]:
                c = self.c.clone().requires_grad_(True)
                f, W = self._weights(c, q)
                v = (W[:, None] * _harmonics(self._scaled(c, q), self.lmax) / self.facl
                     * x[self.b[q]]).sum(1)
                u = torch.where(f <= 1.0, 1.0 - f, torch.zeros_like(f))
                rows = torch.unique(self.row[q])
                value = (wxi[self.row[q]] * v).sum() - (wxi * u * self.phi_grid)[rows].sum()
                grad += torch.autograd.grad(value, c)[0]
            lo = hi
        at, a, _ = self.cavity()
        zeta = fep * (wxi * self.u)[at]
        e, z = self.fields(zeta)
        return (-fep * grad).index_add(0, a, -zeta[:, None] * e) - self.q[:, None] * z, z


def _coulomb(q, src, trg):
    """Potential and field of charges q at src on the points trg."""
    phi, e = torch.zeros_like(trg[:, 0]), torch.zeros_like(trg)
    if not len(src):
        return phi, e
    step = max(1, int(1.5e8) // len(src))
    for k in range(0, len(trg), step):
        d = trg[k:k + step, None] - src[None]
        ir = 1.0 / d.square().sum(2).sqrt()
        phi[k:k + step] = ir @ q
        e[k:k + step] = torch.einsum("tsk,ts->tk", d, ir ** 3 * q)
    return phi, e


def exact(case, seed):
    kind = case["kind"]
    if kind == "charges":
        q, src, trg = (torch.as_tensor(v) for v in _charges(case, seed))
        if torch.cuda.is_available():
            q, src, trg = q.cuda(), src.cuda(), trg.cuda()
        phi, ef = _coulomb(q, src, trg)
        return dict(phi=phi, ef=ef)
    n = case.get("n", 0)
    mols = _batch(case, seed) if kind == "batch" else None
    if mols is not None:
        n = sum(len(m["q"]) for m in mols)
    if n > 8000:
        return None
    P = _Exact(mols or [_solved(case, seed)], case["lmax"], case["ngrid"])
    if P.size > P.MOST:
        return None
    if kind == "operators":
        x, s = (torch.as_tensor(v, device=P.dev) for v in _vectors(case, seed))
        y, z = P.lx(x), P.lstarx(s)
        return {"pair": dict(y=y, z=z), "lx": dict(y=y), "lstarx": dict(z=z)}[case["op"]]
    x, s, e = P.solution()
    fx, e_zeta = P.forces(x, s)
    if kind == "batch":
        return dict(esolv=e, fx=fx)
    out = dict(esolv=e[0], sigma=x, s=s, fx=fx)
    return dict(out, e_zeta=e_zeta) if kind == "staged" else out
