"""Timed cases of the plane-wave DFT path: H*psi on both grids' modes, the
preconditioner, exact exchange, k-points, the band-energy adjoint and a whole
SCF, at the sizes of the configurations and tests of this repository.

Cells are Si diamond (a = 10.26 bohr) and fcc Al (a = 7.65 bohr) with HGH
projectors and seeded displacements; the local potential is a screened
Gaussian-smeared ionic one and the bands are Gaussian noise damped at high
kinetic energy, normalised, as Ritz vectors are.  ``exact`` evaluates the same
operators in 64 bits with torch's FFTs and a direct sum over the projector
points.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from pwdft_develop_b200 import Context

A_SI, A_AL = 10.26, 7.65
_SI = ((0, 0, 0), (0, .5, .5), (.5, 0, .5), (.5, .5, 0),
       (.25, .25, .25), (.25, .75, .75), (.75, .25, .75), (.75, .75, .25))
_AL = ((0, 0, 0), (0, .5, .5), (.5, 0, .5), (.5, .5, 0))
# cell -> (atomic number, valence charge, lattice constant, basis, repetitions)
CELLS = {
    "Al4": (13, 3, A_AL, _AL, (1, 1, 1)),
    "Si8": (14, 4, A_SI, _SI, (1, 1, 1)),
    "Si16": (14, 4, A_SI, _SI, (2, 1, 1)),
    "Al32": (13, 3, A_AL, _AL, (2, 2, 2)),
    "Si64": (14, 4, A_SI, _SI, (2, 2, 2)),
    "Si216": (14, 4, A_SI, _SI, (3, 3, 3)),
}
# grids a cell is used on, and the widest block of bands
USE = {
    "Al4": ((16, 20, 24), 24),
    "Si8": ((20, 24, 30, 32), 64),
    "Si16": (((40, 20, 20), (48, 24, 24)), 128),
    "Al32": ((36, 40, 48, 60), 160),
    "Si64": ((36, 40, 48, 60), 320),
    "Si216": ((72,), 480),
}
# HGH (1998): r_loc, s channel (r, h11, h22), p channel (r, h11); all are cut at 3.5 bohr
HGH = {13: (0.45, (0.460104, 5.088340, 2.679700), (0.536744, 2.193438)),
       14: (0.44, (0.422738, 5.906928, 3.258196), (0.484278, 2.727013))}
RCUT = 3.5
DISPLACE = 0.02
SCF_REL = 1e-5


def listed():
    return [
        # the smallest call: a few bands of a small metal cell, as a Lanczos bound or a restart check makes
        {"name": "hpsi_al4_20_f32", "kind": "hpsi", "cell": "Al4", "n": 20, "nband": 7, "prec": "f32",
         "accumulate": False, "filter": False},
        # one H*psi of the small cell's full block in double, every LOBPCG step
        {"name": "hpsi_si8_24_f64", "kind": "hpsi", "cell": "Si8", "n": 24, "nband": 24, "prec": "f64",
         "accumulate": False, "filter": False},
        # an odd block on the radix-3/5 grid added to an existing block (Spinor::Add*)
        {"name": "hpsi_al32_60_f32", "kind": "hpsi", "cell": "Al32", "n": 60, "nband": 61, "prec": "f32",
         "accumulate": True, "filter": False},
        # the headline sweep: one Chebyshev filter step of the FP32 SCF
        {"name": "hpsi_si64_48_f32", "kind": "hpsi", "cell": "Si64", "n": 48, "nband": 160, "prec": "f32",
         "accumulate": False, "filter": False},
        # the same sweep in double, as the refinement iterations and the plain FP64 SCF run it
        {"name": "hpsi_si64_48_f64", "kind": "hpsi", "cell": "Si64", "n": 48, "nband": 160, "prec": "f64",
         "accumulate": False, "filter": True},
        # the largest block: Si216 with its empty bands
        {"name": "hpsi_si216_72_f32", "kind": "hpsi", "cell": "Si216", "n": 72, "nband": 480, "prec": "f32",
         "accumulate": False, "filter": False},
        # the Teter preconditioner on a residual block (LOBPCG, PPCG, Davidson)
        {"name": "teter_si64_48_f32", "kind": "teter", "cell": "Si64", "n": 48, "nband": 160, "prec": "f32"},
        # a k-point batch: 4 x 4 x 4 Monkhorst-Pack, 24 complex bands each
        {"name": "kbatch_si8_24_f32", "kind": "kbatch", "cell": "Si8", "n": 24, "nband": 24, "mesh": 4, "prec": "f32"},
        # the sphere-cut mode (the reference's default representation)
        {"name": "gspace_si64_96_f32", "kind": "gspace", "cell": "Si64", "n": 96, "ecut": 25.0, "nband": 160,
         "prec": "f32"},
        # PBE0 exchange of a block over all occupied orbitals (one ACE rebuild)
        {"name": "exx_si64_48_f32", "kind": "exx", "cell": "Si64", "n": 48, "nband": 160, "norb": 128, "prec": "f32"},
        # d(band energy)/dV_loc and /dR of the occupied bands
        {"name": "adjoint_si64_48_f64", "kind": "adjoint", "cell": "Si64", "n": 48, "nband": 128, "prec": "f64"},
        # a whole mixed-precision ChebFSI SCF to 1e-6 Ha/atom
        {"name": "scf_si64_48_mixed", "kind": "scf", "cell": "Si64", "n": 48, "ecut": 20.0, "nocc": 128, "nextra": 32,
         "mixed": True},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["hpsi"] * 6 + ["teter", "kbatch", "gspace", "exx", "adjoint", "scf"])
    prec = rng.choice(["f32", "f32", "f64"])
    if kind in ("hpsi", "teter", "adjoint"):
        cell = rng.choice(list(CELLS) if kind == "hpsi" else ["Al4", "Si8", "Si16", "Al32", "Si64"])
        grids, top = USE[cell]
        if cell == "Si216" and prec == "f64":
            top = 160
        c = {"kind": kind, "cell": cell, "n": _plain_grid(rng.choice(grids)),
             "nband": _log(rng, 1 if kind != "adjoint" else 4, top), "prec": prec}
        if kind == "hpsi":
            c["accumulate"] = rng.random() < 0.3
            c["filter"] = not c["accumulate"] and rng.random() < 0.3
        if kind == "adjoint":
            c["prec"] = "f64"
            c["nband"] = min(c["nband"], 160)
        return c
    if kind == "kbatch":
        return {"kind": kind, "cell": "Si8", "n": rng.choice([20, 24, 30]), "nband": rng.randint(8, 32),
                "mesh": rng.choice([1, 2, 3, 4]), "prec": "f32"}
    if kind == "gspace":
        cell, n, e0, e1, top = rng.choice([("Si8", 48, 15.0, 24.0, 48), ("Si64", 80, 12.0, 17.0, 160),
                                           ("Si64", 96, 15.0, 25.0, 160)])
        return {"kind": kind, "cell": cell, "n": n, "ecut": round(rng.uniform(e0, e1), 2),
                "nband": _log(rng, 4, top), "prec": prec}
    if kind == "exx":
        cell, n, top = rng.choice([("Si8", 24, 32), ("Si8", 32, 32), ("Si64", 36, 128), ("Si64", 48, 128)])
        return {"kind": kind, "cell": cell, "n": n, "nband": _log(rng, 2, top if prec == "f32" else top // 2),
                "norb": rng.randint(top // 2, top), "prec": prec}
    n = rng.choice([16, 24])
    return {"kind": "scf", "cell": "Si8", "n": n, "ecut": round(rng.uniform(0.8, 1.0) * (5.0 if n == 16 else 10.0), 2),
            "nocc": 16, "nextra": rng.randint(6, 14), "mixed": rng.random() < 0.5}


def _plain_grid(g):
    """Cubic grids as one number, elongated ones as text (plain values)."""
    return g if isinstance(g, int) else "x".join(str(x) for x in g)


def _grid(n):
    return tuple(int(x) for x in n.split("x")) if isinstance(n, str) else (int(n),) * 3


def _dtype(case):
    return torch.float64 if case.get("prec", "f64") == "f64" else torch.float32


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _atoms(case, seed):
    z, _, a, base, reps = CELLS[case["cell"]]
    rng = np.random.Generator(np.random.Philox(seed))
    cells = np.array([(x, y, w) for w in range(reps[2]) for y in range(reps[1]) for x in range(reps[0])], float)
    pos = ((cells[:, None, :] + np.array(base)[None]) * a).reshape(-1, 3)
    pos = pos + rng.uniform(-DISPLACE, DISPLACE, size=pos.shape)
    return [a * r for r in reps], z, pos


def _freq(n, half=False):
    """Signed frequencies with the Nyquist one at +n/2."""
    k = torch.arange(n, dtype=torch.float64, device="cuda")
    k = torch.where(k > n // 2, k - n, k)
    return k[: n // 2 + 1] if half else k


def _g2(L, n, half=False, k=(0.0, 0.0, 0.0)):
    g = [2 * math.pi / L[d] * _freq(n[d], half and d == 0) + k[d] for d in range(3)]
    return g[2][:, None, None] ** 2 + g[1][None, :, None] ** 2 + g[0][None, None, :] ** 2


def _potential(L, nf, z, pos):
    """Screened, Gaussian-smeared ionic potential on the fine grid (zero mean)."""
    rl, vol, zion = HGH[z][0], L[0] * L[1] * L[2], {13: 3.0, 14: 4.0}[z]
    p = torch.tensor(pos, device="cuda")
    e = [torch.exp(-1j * p[:, d, None] * (2 * math.pi / L[d]) * _freq(nf[d], d == 0)[None, :]) for d in range(3)]
    yz = (e[2][:, :, None] * e[1][:, None, :]).reshape(len(pos), -1)
    s = (yz.T @ e[0]).reshape(nf[2], nf[1], -1)
    g2 = _g2(L, nf, half=True)
    v = -4 * math.pi * zion / vol * torch.exp(-0.5 * g2 * rl * rl) / (g2 + 0.8)
    v[0, 0, 0] = 0
    return (torch.fft.irfftn(s * v, s=(nf[2], nf[1], nf[0])) * (nf[0] * nf[1] * nf[2])).reshape(-1)


def _bands(L, n, nband, seed, dtype, cplx=False):
    """Normalised noise bands (nband, n0 n1 n2) damped at high kinetic energy."""
    g = torch.Generator(device="cuda").manual_seed(int(seed) + 17)
    nt = n[0] * n[1] * n[2]
    ctype = torch.complex128 if dtype == torch.float64 else torch.complex64
    out = torch.empty((nband, nt), dtype=ctype if cplx else dtype, device="cuda")
    damp = (1.0 / (1.0 + 0.5 * _g2(L, n) / 3.0) ** 2).to(dtype)
    for b0 in range(0, nband, 32):
        nb = min(32, nband - b0)
        x = torch.randn((nb, n[2], n[1], n[0], 2), generator=g, device="cuda", dtype=dtype)
        y = torch.fft.ifftn(torch.fft.fftn(torch.view_as_complex(x), dim=(1, 2, 3)) * damp, dim=(1, 2, 3))
        y = y.reshape(nb, nt)
        y = y if cplx else y.real
        out[b0:b0 + nb] = y / torch.linalg.vector_norm(y, dim=1, keepdim=True)
    return out


def _channels(z):
    """Projector channels (l, weight, a) with radial part r^l (a0 + a1 r^2) exp(-r^2 / 2 rl^2)."""
    _, (r0, h11, h22), (r1, p11) = HGH[z]

    def norm(l, i, r):
        ex = l + (4 * i - 1) / 2.0
        return math.sqrt(2.0) / (r ** ex * math.sqrt(math.gamma(ex)))

    h12 = -0.5 * math.sqrt(0.6) * h22
    d, v = np.linalg.eigh(np.array([[h11, h12], [h12, h22]]))
    out = []
    for k in (1, 0):
        u = v[:, k] * np.sign(v[np.argmax(np.abs(v[:, k])), k])
        out.append((0, d[k], r0, (u[0] * norm(0, 1, r0), u[1] * norm(0, 2, r0))))
    out.append((1, p11, r1, (norm(1, 1, r1), 0.0)))
    return out


def _projectors(L, nf, z, pos, grad=False):
    """Per atom (idx, beta [5, npts], displacement [npts, 3], grad [3, 5, npts]), and the 5 weights."""
    h = [L[d] / nf[d] for d in range(3)]
    chan = _channels(z)
    wgt = [c[1] for c in chan[:2]] + [chan[2][1]] * 3
    atoms = []
    for p in pos:
        ax = [torch.arange(math.floor((p[d] - RCUT) / h[d]), math.ceil((p[d] + RCUT) / h[d]) + 1, device="cuda")
              for d in range(3)]
        if any(len(a) > nf[d] for d, a in enumerate(ax)):
            # a sphere as wide as the cell: wrapped points once each, at their nearest image
            ax = [torch.arange(round(float(p[d] / h[d])) - nf[d] // 2 + 1,
                               round(float(p[d] / h[d])) + nf[d] // 2 + 1, device="cuda")
                  if len(a) > nf[d] else a for d, a in enumerate(ax)]
        k, j, i = torch.meshgrid(ax[2], ax[1], ax[0], indexing="ij")
        x = torch.stack([c.reshape(-1).double() * h[d] - p[d] for d, c in enumerate((i, j, k))], 1)
        sel = (x * x).sum(1) < RCUT * RCUT
        x = x[sel]
        i, j, k = i.reshape(-1)[sel] % nf[0], j.reshape(-1)[sel] % nf[1], k.reshape(-1)[sel] % nf[2]
        r2 = (x * x).sum(1)
        beta, gr = [], []
        for l, _, rl, (a0, a1) in chan:
            e = torch.exp(-r2 / (2 * rl * rl))
            f = (a0 + a1 * r2) * e
            df = (2 * a1 - (a0 + a1 * r2) / (rl * rl)) * e          # (df/dr) / r
            if l == 0:
                y = math.sqrt(1 / (4 * math.pi))
                beta.append(y * f)
                gr.append(torch.stack([y * df * x[:, d] for d in range(3)]))
            else:
                y = math.sqrt(3 / (4 * math.pi))
                for c in (2, 0, 1):
                    beta.append(y * f * x[:, c])
                    gr.append(torch.stack([y * (df * x[:, c] * x[:, d] + (f if c == d else 0 * f)) for d in range(3)]))
        atoms.append((i + nf[0] * (j + nf[1] * k), torch.stack(beta), x, torch.stack(gr, 1) if grad else None))
    return atoms, np.array(wgt)


def _fine(n):
    return tuple(2 * x for x in n)


def _mp_mesh(L, m):
    f = [(2 * i - m + 1) / (2.0 * m) for i in range(m)]
    return np.array([[2 * math.pi / L[0] * a, 2 * math.pi / L[1] * b, 2 * math.pi / L[2] * c]
                     for c in f for b in f for a in f])


def _occupations(nb, norb_full):
    return np.array([1.0 if b < norb_full else 0.5 for b in range(nb)])


# sphere-cut mode ------------------------------------------------------------
def _sphere(L, n, ecut):
    """Flat R2C index and Miller indices of the stored half sphere, ascending."""
    m0, m1, m2 = _freq(n[0], True), _freq(n[1]), _freq(n[2])
    M2, M1, M0 = torch.meshgrid(m2, m1, m0, indexing="ij")
    keep = (M0 > 0) | ((M0 == 0) & ((M1 > 0) | ((M1 == 0) & (M2 >= 0))))
    e = 0.5 * _g2(L, n, half=True)
    idx = torch.nonzero((keep & (e < ecut)).reshape(-1)).reshape(-1)
    m = torch.stack([M0.reshape(-1)[idx], M1.reshape(-1)[idx], M2.reshape(-1)[idx]], 1)
    return m, e.reshape(-1)[idx]


def _sphere_projectors(L, z, pos, m):
    """vnlc (ns, nproj) and weights from the closed-form transforms of the HGH radial parts."""
    vol = L[0] * L[1] * L[2]
    g = m * torch.tensor([2 * math.pi / x for x in L], dtype=torch.float64, device="cuda")
    q2 = (g * g).sum(1)
    cols, wgt = [], []
    for l, h, rl, (a0, a1) in _channels(z):
        e = math.sqrt(math.pi / 2) * torch.exp(-0.5 * q2 * rl * rl)
        w = h * (4 * math.pi) ** 2 / vol
        if l == 0:
            v = (a0 * rl ** 3 + a1 * rl ** 5 * (3 - q2 * rl * rl)) * e
            cols.append(math.sqrt(1 / (4 * math.pi)) * v.to(torch.complex128))
            wgt.append(w)
        else:
            for c in (2, 0, 1):
                cols.append(-1j * math.sqrt(3 / (4 * math.pi)) * a0 * rl ** 5 * e * g[:, c])
                wgt.append(w)
    vkb = torch.stack(cols, 1)
    vkb[1:] *= math.sqrt(2.0)
    ph = torch.exp(-1j * (g @ torch.tensor(np.asarray(pos).T, device="cuda")))       # (ns, natom)
    return (ph[:, :, None] * vkb[:, None, :]).reshape(len(m), -1), np.tile(wgt, len(pos))


def _sphere_bands(m, ekin, nband, seed, dtype):
    g = torch.Generator(device="cuda").manual_seed(int(seed) + 17)
    x = torch.randn((nband, len(m), 2), generator=g, device="cuda", dtype=dtype)
    x = x / ((1.0 + ekin / 3.0) ** 2).to(dtype)[None, :, None]
    x[:, 0, 1] = 0
    x = x.reshape(nband, -1)
    return (x / torch.linalg.vector_norm(x, dim=1, keepdim=True)).contiguous()


# ---------------------------------------------------------------------------
# the measured calls
# ---------------------------------------------------------------------------
def prepare(case, seed):
    kind, n = case["kind"], _grid(case["n"])
    L, z, pos = _atoms(case, seed)
    prec = case.get("prec", "f64")
    dtype = _dtype(case)
    s = {"kind": kind}
    if kind == "gspace":
        c = Context.gspace(L, n, case["ecut"], precision=prec)
        m, ekin = _sphere(L, n, case["ecut"])
        v, w = _sphere_projectors(L, z, pos, m)
        c.gs_set_projectors(v.cpu().numpy(), w)
        c.set_vtot(_potential(L, n, z, pos).cpu().numpy())
        s["psi"] = _sphere_bands(m, ekin, case["nband"], seed, dtype)
        s["ctx"] = c
        return s
    nf = _fine(n)
    c = Context(L, n, nf, precision=prec)
    s["ctx"] = c
    if kind == "scf":
        c.set_atoms([z] * len(pos), pos)
        s["args"] = dict(nocc=case["nocc"], nextra=case["nextra"], ecut=case["ecut"], solver="chebfsi",
                         mixed=case["mixed"], cheby_degree=10, cheby_first_cycles=5, tol_efree=1e-6,
                         refine_threshold=3e-6, max_iter=60, seed=int(seed) % 100000 + 1, graphs=True)
        return s
    if kind in ("hpsi", "kbatch", "adjoint"):
        c.set_vtot(_potential(L, nf, z, pos).cpu().numpy())
    if kind == "hpsi":
        atoms, w = _projectors(L, nf, z, pos)
        c.set_nonlocal([(i.cpu().numpy(), b.cpu().numpy(), w) for i, b, _, _ in atoms])
        if case["filter"]:
            c.set_wfn_filter(_filter_ecut(L, n))
    elif kind in ("kbatch", "adjoint"):
        c.set_atoms([z] * len(pos), pos)
    if kind == "kbatch":
        k = _mp_mesh(L, case["mesh"])
        c.set_kpoints(k)
        s["psi"] = _bands(L, n, len(k) * case["nband"], seed, dtype, cplx=True).reshape(len(k), case["nband"], -1)
        return s
    s["psi"] = _bands(L, n, case["nband"], seed, dtype)
    if kind == "hpsi" and case["accumulate"]:
        s["a3"] = _bands(L, n, case["nband"], seed + 1, dtype)
    if kind == "exx":
        c.exx_setup(fraction=0.25, screen_mu=0.0, divergence_type=1, ecut=_filter_ecut(L, n))
        c.exx_set_phi(_bands(L, n, case["norb"], seed + 2, dtype), _occupations(case["norb"], case["norb"] - 4))
    if kind == "adjoint":
        s["w"] = 2.0 * _occupations(case["nband"], max(1, case["nband"] - 4))
    return s


def _filter_ecut(L, n):
    """The cut-off a grid is built for: sqrt(2 Ecut) L / pi points per direction, a little inside."""
    return 0.75 * min(0.5 * (math.pi * n[d] / L[d]) ** 2 for d in range(3))


def run(s):
    c, kind = s["ctx"], s["kind"]
    if kind == "hpsi":
        if "a3" in s:
            return c.hpsi(s["psi"], out=s["a3"].clone(), accumulate=True)
        return c.hpsi(s["psi"])
    if kind == "gspace":
        return c.hpsi(s["psi"])
    if kind == "teter":
        return c.teter(s["psi"])
    if kind == "kbatch":
        return c.hpsi_kbatch(s["psi"])
    if kind == "exx":
        return c.exx_apply(s["psi"])
    if kind == "adjoint":
        return c.band_energy_backward(s["psi"], s["w"])
    res, eig, rho = c.scf(**s["args"])
    return {"efree": res["efree"], "eig": eig, "rho": rho}


# ---------------------------------------------------------------------------
# sizes and tolerances
# ---------------------------------------------------------------------------
def _fft(n, lines):
    return 5.0 * n * math.log2(n) * lines


def _hpsi_flops(n, fields, nband, atoms_pts, per=4):
    """Pruned C2C transforms of `fields` complex fields (to the fine grid and back) and the projector sums."""
    nf = _fine(n)
    coarse = _fft(n[0], n[1] * n[2]) + _fft(n[1], n[0] * n[2]) + _fft(n[2], n[0] * n[1])
    fine = _fft(nf[2], n[0] * n[1]) + _fft(nf[1], n[0] * nf[2]) + _fft(nf[0], nf[1] * nf[2])
    return fields * (2 * coarse + 2 * fine + 2.0 * nf[0] * nf[1] * nf[2]) + per * 5.0 * atoms_pts * nband


def work(case):
    kind, n = case["kind"], _grid(case["n"])
    z, _, a, base, reps = CELLS[case["cell"]]
    L = [a * r for r in reps]
    natom = len(base) * reps[0] * reps[1] * reps[2]
    nt, e = n[0] * n[1] * n[2], 8 if case.get("prec", "f64") == "f64" else 4
    vol = L[0] * L[1] * L[2]
    if kind == "gspace":
        ns = vol * (2 * case["ecut"]) ** 1.5 / (12 * math.pi ** 2)     # half sphere
        nb, h = case["nband"], [x // 2 for x in n]
        fields = (nb + 1) // 2
        f = fields * 2 * (_fft(n[2], 0.79 * h[0] * h[1]) + _fft(n[1], h[0] * n[2]) + _fft(n[0], n[1] * n[2]))
        # separable structure factors make the projectors cheap to hold: the dense products are the work
        return {"bytes": e * (4 * ns * nb + nt + 2 * ns * 5 * natom), "flops": f + 2.0 * fields * nt + 8.0 * ns * 5 * natom * nb}
    nf = _fine(n)
    ntf = 8 * nt
    pts = natom * min(ntf, 4.0 / 3.0 * math.pi * RCUT ** 3 * ntf / vol)
    table = pts * (5 * e + 4)
    if kind == "teter":
        nb = case["nband"]
        f = (nb + 1) // 2 * 2 * (_fft(n[0], n[1] * n[2]) + _fft(n[1], n[0] * n[2]) + _fft(n[2], n[0] * n[1]))
        return {"bytes": e * nt * (2 * nb + 1), "flops": f + 2.0 * nt * nb}
    if kind == "exx":
        nb, no = case["nband"], case["norb"]
        one = 2 * (_fft(n[0], n[1] * n[2]) + _fft(n[1], n[0] * n[2]) + _fft(n[2], n[0] * n[1])) + 8.0 * nt
        return {"bytes": e * nt * (2 * nb + no + 1), "flops": nb * ((no + 1) // 2) * one}
    if kind == "kbatch":
        nk = case["mesh"] ** 3
        nb = nk * case["nband"]
        return {"bytes": e * (4 * nt * nb + ntf + nk * nt) + table, "flops": _hpsi_flops(n, nb, nb, pts, per=8)}
    if kind == "scf":
        nb = case["nocc"] + case["nextra"]
        # about 5 + 16 filter passes of degree 10 over all bands, and 17 densities
        sweeps = 5 * 10 + 16 * 11
        return {"bytes": sweeps * (4 * nt * (2 * nb) + 4 * ntf + pts * 24),
                "flops": sweeps * _hpsi_flops(n, (nb + 1) // 2, nb, pts)}
    nb = case["nband"]
    fields = (nb + 1) // 2
    if kind == "adjoint":
        return {"bytes": e * nt * nb + 8 * ntf + pts * (20 * e + 4),
                "flops": 0.5 * _hpsi_flops(n, fields, 0, pts) + 2.0 * 20 * pts * nb}
    return {"bytes": e * (nt * nb * (3 if case["accumulate"] else 2) + ntf) + table,
            "flops": _hpsi_flops(n, fields, nb, pts)}


def tolerance(case):
    """About four times the distance from the 64-bit values (H*psi in FP32 1.0-1.9e-6, set by the
    split-bf16 projector products; transforms alone 1.1-1.9e-7; FP64 1-2e-15, d/dR 1.5e-14)."""
    kind = case["kind"]
    if kind == "scf":
        # converged to 1e-6 Ha/atom in E_free, second order in bands and density: other roundings of the
        # FP32 iterations move the eigenvalues and the density by up to 2.1e-6
        return {"rel": SCF_REL}
    if kind == "adjoint":
        return {"rel": 1e-13}
    if case["prec"] == "f64":
        return {"rel": 1e-14}
    return {"rel": 8e-7 if kind in ("teter", "exx") else 6e-6}


# ---------------------------------------------------------------------------
# 64-bit evaluation
# ---------------------------------------------------------------------------
class _Maps:
    """Coarse -> fine spectrum placement: flat "+" and "-" targets of every coarse coefficient."""

    def __init__(self, n):
        nf = _fine(n)
        k, j, i = torch.meshgrid(*[torch.arange(n[d], device="cuda") for d in (2, 1, 0)], indexing="ij")
        plus, minus, nyq = 0, 0, torch.zeros_like(i, dtype=torch.bool)
        for d, (x, stride) in enumerate(((i, 1), (j, nf[0]), (k, nf[0] * nf[1]))):
            h = n[d] // 2
            p = torch.where(x <= h, x, x + nf[d] - n[d])
            plus = plus + p * stride
            minus = minus + torch.where(x == h, nf[d] - h, p) * stride
            nyq |= x == h
        self.n, self.nf = n, nf
        self.plus, self.minus, self.nyq = plus.reshape(-1), minus.reshape(-1), nyq.reshape(-1)
        self.half = torch.where(self.nyq, 0.5, 1.0).to(torch.float64)

    def up(self, X, cplx=False):
        """Coarse spectrum (nb, N_c), of fftn / N_c, to the fine grid's values."""
        F = torch.zeros((X.shape[0], self.nf[0] * self.nf[1] * self.nf[2]), dtype=X.dtype, device=X.device)
        if cplx:
            F[:, self.plus] = X
        else:
            F[:, self.plus] = X * self.half
            F[:, self.minus[self.nyq]] = X[:, self.nyq] * 0.5
        F = F.reshape(-1, self.nf[2], self.nf[1], self.nf[0])
        return torch.fft.ifftn(F, dim=(1, 2, 3), norm="forward").reshape(X.shape[0], -1)

    def down(self, y, cplx=False):
        """Fine-grid values to the coarse spectrum (of fftn / N_f)."""
        F = torch.fft.fftn(y.reshape(-1, self.nf[2], self.nf[1], self.nf[0]), dim=(1, 2, 3), norm="forward")
        F = F.reshape(y.shape[0], -1)
        if cplx:
            return F[:, self.plus]
        X = F[:, self.plus] * self.half
        X[:, self.nyq] += 0.5 * F[:, self.minus[self.nyq]]
        return X

    def spectrum(self, x):
        n = self.n
        return torch.fft.fftn(x.reshape(-1, n[2], n[1], n[0]), dim=(1, 2, 3), norm="forward").reshape(x.shape[0], -1)

    def values(self, X):
        n = self.n
        return torch.fft.ifftn(X.reshape(-1, n[2], n[1], n[0]), dim=(1, 2, 3), norm="forward").reshape(X.shape[0], -1)


def _pairs(psi):
    """Bands two by two as complex fields in 64 bits."""
    p = psi.double()
    if p.shape[0] % 2:
        p = torch.cat([p, torch.zeros_like(p[:1])])
    return torch.complex(p[0::2], p[1::2])


def _unpair(z, nb):
    return torch.stack([z.real, z.imag], 1).reshape(-1, z.shape[1])[:nb]


def exact(case, seed):
    kind, n = case["kind"], _grid(case["n"])
    if kind == "scf":
        return None
    L, z, pos = _atoms(case, seed)
    vol, nt, nb = L[0] * L[1] * L[2], n[0] * n[1] * n[2], case["nband"]
    dtype = _dtype(case)
    step = max(1, (1 << 26) // (8 * nt))
    if kind == "gspace":
        return _exact_gspace(case, seed, L, z, pos, n, dtype)
    psi = None if kind == "kbatch" else _bands(L, n, nb, seed, dtype)
    m = _Maps(n)
    if kind == "teter":
        a = _g2(L, n).reshape(-1)
        b = 27.0 + a * (18.0 + a * (12.0 + a * 8.0))
        t = b / (b + 16.0 * a ** 4)
        return torch.cat([_unpair(m.values(m.spectrum(Z) * t), 2 * len(Z))
                          for Z in torch.split(_pairs(psi), 8 * step)])[:nb].cpu().numpy()
    if kind == "exx":
        return _exact_exx(case, seed, L, n, m, psi, vol, step)
    nf = _fine(n)
    ntf = 8 * nt
    v = _potential(L, nf, z, pos)
    atoms, w = _projectors(L, nf, z, pos, grad=kind == "adjoint")
    w = torch.tensor(w, device="cuda") * (vol / ntf)
    if kind == "kbatch":
        out = []
        ks = _mp_mesh(L, case["mesh"])
        psi = _bands(L, n, len(ks) * nb, seed, dtype, cplx=True).reshape(len(ks), nb, -1)
        for k, x in zip(ks, psi):
            kt = torch.tensor(k, device="cuda")
            X = m.spectrum(x.to(torch.complex128))
            f = m.up(X, cplx=True)
            u = f * v
            for idx, beta, d, _ in atoms:
                ph = torch.exp(1j * (d @ kt))
                c = ((f[:, idx] * ph) @ beta.T.to(f.dtype)) * w
                u[:, idx] += (c @ beta.to(f.dtype)) * ph.conj()
            out.append(m.values(X * (0.5 * _g2(L, n, k=k)).reshape(-1) + m.down(u, cplx=True)))
        return torch.stack(out).cpu().numpy()
    if kind == "adjoint":
        wb = torch.tensor(2.0 * _occupations(nb, max(1, nb - 4)), device="cuda")
        dv = torch.zeros(ntf, dtype=torch.float64, device="cuda")
        dr = torch.zeros((len(pos), 3), dtype=torch.float64, device="cuda")
        for b0 in range(0, nb, 2 * step):
            p = psi[b0:b0 + 2 * step]
            f = _unpair(m.up(m.spectrum(_pairs(p))), len(p))
            ww = wb[b0:b0 + len(p)]
            dv += (ww @ (f * f)) * (nt / ntf)
            for a, (idx, beta, _, gr) in enumerate(atoms):
                fa = f[:, idx]
                val = (fa @ beta.T) * w
                for d in range(3):
                    dr[a, d] -= 2 * (nt / ntf) * (ww @ (val * (fa @ gr[d].T))).sum()
        return dv.cpu().numpy(), dr.cpu().numpy()
    ek = 0.5 * _g2(L, n).reshape(-1)
    keep = (ek <= _filter_ecut(L, n)).double() if case["filter"] else 1.0
    out = []
    for Z in torch.split(_pairs(psi), step):
        X = m.spectrum(Z)
        f = m.up(X)
        u = f * v
        for idx, beta, _, _ in atoms:
            bc = beta.to(f.dtype)
            u[:, idx] += ((f[:, idx] @ bc.T) * w) @ bc
        out.append(_unpair(m.values((X * ek + m.down(u)) * keep), 2 * len(Z)))
    r = torch.cat(out)[:nb]
    if case["accumulate"]:
        r += _bands(L, n, nb, seed + 1, dtype).double()
    return r.cpu().numpy()


def _exact_exx(case, seed, L, n, m, psi, vol, step):
    nt, no = psi.shape[1], case["norb"]
    occ = _occupations(no, no - 4)
    phi = _bands(L, n, no, seed + 2, dtype=psi.dtype).double() * math.sqrt(nt / vol)
    q = _g2(L, n).reshape(-1)
    alpha = 10.0 / (2.0 * _filter_ecut(L, n))
    big = q > 1e-8
    div = 4 * math.pi * (float((torch.exp(-alpha * q[big]) / q[big]).sum()) - alpha)
    div -= vol / math.sqrt(alpha * math.pi)
    kern = torch.where(big, 4 * math.pi / torch.where(big, q, torch.ones_like(q)), torch.full_like(q, -div))
    out = torch.zeros(psi.shape, dtype=torch.float64, device="cuda")
    p = psi.double()
    for b in range(len(p)):
        for j0 in range(0, no, 32 * step):
            ph = phi[j0:j0 + 32 * step]
            o = torch.tensor(occ[j0:j0 + len(ph)], device="cuda")
            y = _unpair(m.values(m.spectrum(_pairs(p[b] * ph)) * kern), len(ph))
            out[b] -= 0.25 * (o @ (ph * y))
    return out.cpu().numpy()


def _exact_gspace(case, seed, L, z, pos, n, dtype):
    mi, ekin = _sphere(L, n, case["ecut"])
    nb, N = case["nband"], n[0] * n[1] * n[2]
    x = _sphere_bands(mi, ekin, nb, seed, dtype).double()
    c = torch.view_as_complex(x.reshape(nb, -1, 2))
    vnl, w = _sphere_projectors(L, z, pos, mi)
    v = _potential(L, n, z, pos)
    mi = mi.long()
    flat = [(s * mi[:, 0]) % n[0] + n[0] * (((s * mi[:, 1]) % n[1]) + n[1] * ((s * mi[:, 2]) % n[2])) for s in (1, -1)]
    out = c * ekin + ((c @ vnl.conj()).real * torch.tensor(w, device="cuda")).to(c.dtype) @ vnl.T
    f = torch.full((len(mi),), math.sqrt(0.5), dtype=torch.float64, device="cuda")
    f[0] = 1.0
    for b0 in range(0, nb, 16):
        a = c[b0:b0 + 16] * f
        F = torch.zeros((len(a), N), dtype=c.dtype, device="cuda")
        F[:, flat[1]] = a.conj()
        F[:, flat[0]] = a
        r = torch.fft.ifftn(F.reshape(-1, n[2], n[1], n[0]), dim=(1, 2, 3), norm="forward").real
        Y = torch.fft.fftn((r * v.reshape(n[2], n[1], n[0])).to(c.dtype), dim=(1, 2, 3), norm="forward").reshape(len(a), -1)
        out[b0:b0 + 16] += Y[:, flat[0]] / f
    return torch.view_as_real(out.contiguous()).reshape(nb, -1).cpu().numpy()
