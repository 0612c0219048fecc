"""Performance cases of the plane-wave Hamiltonian, density and Davidson paths.

Each case is one call, or one short chain of calls, as a self-consistent-field
program makes it: H|psi> on a block of bands (FP64, mixed, complex64 and
Gamma-only forms), the ultrasoft S|psi>, the charge density of a band block, and
band solves at one k-point followed by their density.  Sizes run from the
two-atom FCC cell to the 128-atom cubic cell of the benchmark configurations.

Inputs are made here from the seed alone: atoms on a jittered grid, Gaussian
wells plus a random smooth field, two s and two p projectors per atom with
coupled D blocks, and bands that fall off with the kinetic energy as
wavefunctions do.  `exact` restates each path in plain torch, in 64 bits.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from q3_b200._lib import FP64, MIXED
from q3_b200.applicator import PlanewaveHamiltonianApplicator
from q3_b200.davidson import PlanewaveDavidsonDiagonalizer

DEVICE = "cuda"
PROJECTORS_PER_ATOM = 8  # two s, two p
# FFT lengths in use for cells of up to 128 atoms
GRIDS = (24, 25, 27, 30, 32, 36, 40, 45, 48, 50, 54, 60, 64, 72, 75, 80, 90, 96, 100, 108)


def _case(kind, atoms, ecut, bands, a=0.0, precision="fp64", fcc=False, k=0.0, iterations=0, grid=0, **more):
    """`a` 0: the lattice constant of the serving cells, 5.13 atoms^(1/3) bohr; `grid` 0: the
    smallest length that holds products of two bands; k: the k-point k (1, 1, 2) / 1."""
    a = a or 5.13 * atoms ** (1.0 / 3.0)
    if not grid:
        need = 4.0 * math.sqrt(ecut) * a / (2.0 * math.pi) + 1.0
        grid = next(n for n in GRIDS if n >= need or n == GRIDS[-1])
    return {"kind": kind, "atoms": atoms, "ecut": ecut, "bands": bands, "a": a, "grid": grid, "fcc": fcc, "k": k,
            "precision": precision, "iterations": iterations, **more}


def listed():
    return [
        # the two-atom FCC cell: the smallest call a solver makes, all latency and launches
        _case("hpsi", 2, 30.0, 8, a=10.26, fcc=True, grid=24, name="hpsi_2atoms_fp64"),
        # one k-point of the eight-atom cell with a shifted 4x4x2 mesh: the ordinary small cell
        _case("hpsi", 8, 30.0, 48, a=10.26, grid=40, k=0.125, name="hpsi_8atoms_fp64"),
        # a request of the serving stream: odd atom and band counts, FP32 inside, FP64 vectors
        _case("hpsi", 19, 33.7, 77, precision="mixed", name="hpsi_19atoms_mixed"),
        # the 64-atom throughput cell in plain FP64, and in FP32 as a mixed solve applies it
        _case("hpsi", 64, 30.0, 256, a=20.5, grid=80, name="hpsi_64atoms_fp64"),
        _case("hpsi", 64, 30.0, 256, a=20.5, grid=80, precision="c64", name="hpsi_64atoms_c64"),
        # the largest cell: 128 atoms, 512 bands, 1024 projectors
        _case("hpsi", 128, 36.0, 512, a=25.8, grid=108, name="hpsi_128atoms_fp64"),
        # Gamma-only sampling of a large cell: half-sphere vectors, an odd band left unpaired
        _case("gamma", 32, 30.0, 129, name="gamma_32atoms_fp64"),
        # the ultrasoft overlap on the block of unconverged bands
        _case("overlap", 64, 30.0, 90, a=20.5, grid=80, name="overlap_64atoms_fp64"),
        # the charge density of all bands after a solve, a few of them empty
        _case("density", 64, 30.0, 256, a=20.5, grid=80, name="density_64atoms"),
        # a converged k-point of the eight-atom cell, and its density
        _case("solve", 8, 30.0, 48, a=10.26, grid=40, k=0.125, name="solve_8atoms_fp64"),
        # the same kind of cell served in mixed precision
        _case("solve", 6, 30.0, 24, precision="mixed", name="solve_6atoms_mixed"),
        # a few Davidson steps of the 64-atom cell, as one SCF cycle takes them
        _case("solve", 64, 30.0, 256, a=20.5, grid=80, iterations=6, name="steps_64atoms_fp64"),
    ]


def draw(rng):
    def between(lo, hi):
        return math.exp(rng.uniform(math.log(lo), math.log(hi)))

    kind = rng.choice(["hpsi", "hpsi", "hpsi", "gamma", "overlap", "density", "solve"])
    small = kind == "solve"
    atoms = int(between(2, 13 if small else 97))
    ecut = round(rng.uniform(20.0, 30.0 if small else 36.0), 3)
    bands = max(5, int(atoms * rng.uniform(2.0, 4.5))) if not small else 4 * atoms
    precision = rng.choice(["fp64", "fp64", "mixed", "c64"] if kind == "hpsi" else
                           ["fp64", "mixed"] if kind in ("gamma", "overlap", "solve") else ["fp64"])
    iterations = 6 if small and rng.random() < 0.3 else 0
    return _case(kind, atoms, ecut, bands, precision=precision, k=0.0 if kind == "gamma" else
                 rng.choice([0.0, 0.125, round(rng.uniform(0.0, 0.5), 3)]), iterations=iterations)


# ------------------------------------------------------------------ inputs

def _lattice(c):
    if c["fcc"]:
        return 0.5 * c["a"] * np.array([[0.0, 1.0, 1.0], [1.0, 0.0, 1.0], [1.0, 1.0, 0.0]])
    return c["a"] * np.eye(3)


def _waves(c):
    """Miller indices, |k+G|^2 (Ry) and k+G of the sphere, by rising energy."""
    rec = 2.0 * np.pi * np.linalg.inv(_lattice(c)).T
    most = [int(math.ceil(math.sqrt(c["ecut"]) * np.linalg.norm(v) / (2.0 * np.pi))) + 2 for v in _lattice(c)]
    mil = np.array(np.meshgrid(*[np.arange(-m, m + 1) for m in most], indexing="ij")).reshape(3, -1).T
    q = (mil + c["k"] * np.array([1.0, 1.0, 2.0])) @ rec
    ke = np.einsum("ij,ij->i", q, q)
    keep = np.flatnonzero(ke <= c["ecut"])
    keep = keep[np.argsort(ke[keep], kind="stable")]
    mil, ke, q = mil[keep], ke[keep], q[keep]
    if c["kind"] == "gamma":  # the half sphere, the origin first
        lead = np.where(mil[:, 0] != 0, mil[:, 0], np.where(mil[:, 1] != 0, mil[:, 1], mil[:, 2]))
        half = np.concatenate([np.flatnonzero(np.all(mil == 0, axis=1)), np.flatnonzero(lead > 0)])
        mil, ke, q = mil[half], ke[half], q[half]
    return mil, ke, q


def _on_grid(mil, n):
    w = np.where(mil < 0, mil + n, mil)
    return ((w[:, 0] * n + w[:, 1]) * n + w[:, 2]).astype(np.int32)


def _inputs(c, seed):
    g = torch.Generator(device=DEVICE)
    g.manual_seed(int(seed))
    rng = np.random.default_rng(int(seed))
    n, na, nb = c["grid"], c["atoms"], c["bands"]
    mil, ke, q = _waves(c)
    lat = _lattice(c)
    vol = abs(np.linalg.det(lat))
    side = int(math.ceil(na ** (1.0 / 3.0) - 1e-9))
    sites = np.array(np.meshgrid(*[np.arange(side)] * 3, indexing="ij")).reshape(3, -1).T[:na]
    frac = (sites + 0.5 + rng.uniform(-0.2, 0.2, (na, 3))) / side
    # V(r): wells of -4 Ry and sigma 1 bohr, and a smooth field of 0.1 Ry a component below 3 / bohr
    m1 = np.arange(n)
    m1 = np.where(m1 <= n // 2, m1, m1 - n)
    rec = torch.from_numpy(2.0 * np.pi * np.linalg.inv(lat).T).to(DEVICE)
    mm = torch.from_numpy(m1.astype(np.float64)).to(DEVICE)
    G = (mm[:, None, None, None] * rec[0] + mm[None, :, None, None] * rec[1] + mm[None, None, :, None] * rec[2])
    g2 = (G * G).sum(-1)
    ph = [torch.polar(torch.ones(na, n, dtype=torch.float64, device=DEVICE),
                      -2.0 * math.pi * torch.from_numpy(frac[:, d:d + 1]).to(DEVICE) * mm) for d in range(3)]
    sf = torch.einsum("ai,aj,ak->ijk", ph[0], ph[1], ph[2])
    noise = torch.randn(n, n, n, dtype=torch.float64, device=DEVICE, generator=g)
    vg = -4.0 * (2.0 * math.pi) ** 1.5 / vol * torch.exp(-0.5 * g2) * sf
    vg = vg + torch.where(g2 < 9.0, 0.1 / math.sqrt(n ** 3) * torch.fft.fftn(noise), 0.0)
    v = torch.fft.ifftn(vg).real * n ** 3
    # projectors: two s and two p per atom, widths 1.5 and 1.1 bohr
    qt = torch.from_numpy(q).to(DEVICE)
    q2 = torch.from_numpy(ke).to(DEVICE)
    shapes = []
    for w in (1.5, 1.1):
        shapes.append(math.pi ** 1.5 * w ** 3 / math.sqrt(4 * math.pi) * torch.exp(-0.25 * q2 * w * w) + 0j)
    for w in (1.5, 1.1):
        f = 0.5 * math.pi ** 1.5 * w ** 5 * math.sqrt(3.0 / (4.0 * math.pi)) * torch.exp(-0.25 * q2 * w * w)
        shapes += [-1j * f * qt[:, d] for d in range(3)]
    shapes = torch.stack(shapes)                                            # 8 x npw
    tau = torch.from_numpy(frac @ lat).to(DEVICE)
    phase = torch.polar(torch.full((na, len(ke)), vol ** -0.5, dtype=torch.float64, device=DEVICE), -(tau @ qt.T))
    beta = (phase[:, None, :] * shapes[None]).reshape(na * PROJECTORS_PER_ATOM, -1)  # P x npw

    def block(scale):  # couples the two channels of each (l, m)
        s, p = rng.uniform(-scale, scale, (2, 2)), rng.uniform(-scale, scale, (2, 2))
        b = np.zeros((8, 8))
        b[:2, :2] = 0.5 * (s + s.T)
        for d in range(3):
            b[np.ix_([2 + d, 5 + d], [2 + d, 5 + d])] = 0.5 * (p + p.T)
        return b

    dmat, qmat = block(2.0), block(0.3)
    psi = torch.randn(nb, len(ke), dtype=torch.complex128, device=DEVICE, generator=g) / (1.0 + q2)
    if c["kind"] == "gamma":
        psi[:, 0] = psi[:, 0].real + 0j
    if c["kind"] == "solve":
        psi = torch.linalg.qr(psi.T)[0].T.contiguous()
    psi = psi / torch.linalg.vector_norm(psi, dim=1, keepdim=True)
    if c["precision"] == "c64":
        psi = psi.to(torch.complex64)
    occupied = nb - nb // 8
    wts = np.where(np.arange(nb) < occupied, 2.0 / vol, 0.0)
    return {"mil": mil, "ke": ke, "v": v, "beta": beta, "d": dmat, "q": qmat, "psi": psi, "weights": wts,
            "occupied": occupied}


def prepare(case, seed):
    c, n = case, case["grid"]
    x = _inputs(c, seed)
    ap = PlanewaveHamiltonianApplicator(device=0)
    ap.update_potential(x["v"].cpu().numpy(), (n, n, n))
    beta = np.asfortranarray(x["beta"].cpu().numpy().T)
    offs = np.arange(0, beta.shape[1] + 1, PROJECTORS_PER_ATOM, dtype=np.int32)
    blocks = np.tile(x["d"].reshape(-1, order="F"), c["atoms"])
    g2g = _on_grid(x["mil"], n)
    if c["kind"] == "gamma":
        ap.prepare_kpoint_gamma(len(g2g), g2g, _on_grid(-x["mil"], n), x["ke"], beta, offs, blocks)
    else:
        ap.prepare_kpoint(0, len(g2g), g2g, x["ke"], beta, offs, blocks)
    s = {"kind": c["kind"], "ap": ap, "psi": x["psi"], "nb": c["bands"], "weights": x["weights"],
         "precision": MIXED if c["precision"] == "mixed" else FP64}
    if c["kind"] == "overlap":
        ap.set_overlap_blocks(np.tile(x["q"].reshape(-1, order="F"), c["atoms"]))
    if c["kind"] in ("density", "solve"):
        s["rho"] = torch.zeros(n ** 3, dtype=torch.float64, device=DEVICE)
    if c["kind"] == "solve":
        dv = PlanewaveDavidsonDiagonalizer(ap, s["precision"])
        dv.set_occupied_bands(x["occupied"])
        dv.set_tolerance(1e-9)
        dv.set_maximum_iterations(c["iterations"] or 200)
        s["solver"] = dv
    s["out"] = torch.empty_like(x["psi"])
    return s


def run(s):
    kind, ap, psi, out, nb = s["kind"], s["ap"], s["psi"], s["out"], s["nb"]
    if kind == "hpsi":
        ap.apply_batch(psi, out, nb, s["precision"])
    elif kind == "gamma":
        ap.apply_batch_gamma(psi, out, nb, s["precision"])
    elif kind == "overlap":
        ap.apply_overlap(psi, out, nb, s["precision"])
    elif kind == "density":
        ap.accumulate_density(psi, s["weights"], s["rho"].zero_())
        return s["rho"]
    else:
        out.copy_(psi)  # the solve works in place
        r = s["solver"].solve(out, nb)
        ap.accumulate_density(out, s["weights"], s["rho"].zero_())
        return {"eigenvalues": r.eigenvalues, "density": s["rho"]}
    return out


# ------------------------------------------------------------------ what a pass cannot do without

def work(case):
    c = case
    rec = 2.0 * math.pi / c["a"]
    npw = c["ecut"] ** 1.5 * 4.0 * math.pi / 3.0 / rec ** 3 * (0.25 if c["fcc"] else 0.5 if c["kind"] == "gamma" else 1.0)
    P, nb, N = PROJECTORS_PER_ATOM * c["atoms"], c["bands"], c["grid"] ** 3
    cb = 8 if c["precision"] == "c64" else 16
    # the transform pair of one band: the lines along the first axis that hold the sphere, half
    # the rows of the second, all of the third (0.565 of a full 5 N log2 N each way)
    fft = 2 * 0.565 * 5.0 * N * math.log2(N)
    inside = 8 if c["precision"] in ("c64", "mixed") else 16  # bytes of a projector entry as used
    vectors, table = 2 * npw * nb * cb, npw * P * inside
    if c["kind"] == "density":
        return {"bytes": npw * nb * 16 + 16.0 * N, "flops": 0.5 * fft * c["bands"] + 3.0 * N * nb}
    if c["kind"] == "overlap":
        return {"bytes": vectors + table, "flops": 16.0 * npw * P * nb}
    columns = (nb + 1) // 2 if c["kind"] == "gamma" else nb  # two bands ride one transform
    h = {"bytes": vectors + table + 8.0 * N + 8.0 * npw, "flops": columns * fft + 16.0 * npw * P * nb}
    if c["kind"] != "solve":
        return h
    # a Davidson step: H on the block; projection, Cholesky-QR, the two subspace rows, residuals and
    # the collapse as complex products of npw x nb by the basis (at most 2 nb columns)
    steps = c["iterations"] or 20
    gemm = 8.0 * npw * nb * nb
    return {"bytes": steps * (h["bytes"] + 6 * npw * nb * 16), "flops": steps * (h["flops"] + 12 * gemm)}


def tolerance(case):
    if case["kind"] == "solve":
        # a solve to 1e-9 Ry in the occupied eigenvalues leaves the empty bands at 1e-5 Ry, 1e-6 of the
        # eigenvalues' norm (1.2e-6 against the dense eigensolver), and the density within 6e-7 of it
        return {"rel": 1e-5, "max": 1e-3}
    if case["precision"] in ("c64", "mixed"):
        return {"rel": 1e-5, "max": 4e-4}  # 2e-6 seen against 64 bits
    return {"rel": 2e-15, "max": 2e-13}    # 1e-16 to 4e-16 seen


# ------------------------------------------------------------------ the same in plain torch, 64 bits

def _chunks(nb, n):
    per = max(1, int(1.5e9 / (16.0 * n ** 3)))
    return [slice(i, min(nb, i + per)) for i in range(0, nb, per)]


def _apply(x, n, psi, mil=None, ke=None, beta=None):
    """H psi of rows of full-sphere vectors."""
    mil = x["mil"] if mil is None else mil
    ke = torch.from_numpy(x["ke"] if ke is None else ke).to(DEVICE)
    beta = x["beta"] if beta is None else beta
    at = torch.from_numpy(_on_grid(mil, n).astype(np.int64)).to(DEVICE)
    out = ke * psi
    for s in _chunks(len(psi), n):
        grid = torch.zeros(len(psi[s]), n ** 3, dtype=torch.complex128, device=DEVICE)
        grid[:, at] = psi[s]
        r = torch.fft.ifftn(grid.view(-1, n, n, n), dim=(1, 2, 3)) * x["v"]
        out[s] += torch.fft.fftn(r, dim=(1, 2, 3)).reshape(len(grid), -1)[:, at]
    return out + _nonlocal(beta, x["d"], psi)


def _nonlocal(beta, blocks, psi):
    b = (psi @ beta.conj().T).view(len(psi), -1, PROJECTORS_PER_ATOM)
    d = torch.from_numpy(blocks).to(DEVICE).to(torch.complex128)
    return torch.einsum("vaj,ij->vai", b, d).reshape(len(psi), -1) @ beta


def _density(x, n, psi):
    at = torch.from_numpy(_on_grid(x["mil"], n).astype(np.int64)).to(DEVICE)
    w = torch.from_numpy(x["weights"]).to(DEVICE)
    rho = torch.zeros(n ** 3, dtype=torch.float64, device=DEVICE)
    for s in _chunks(len(psi), n):
        grid = torch.zeros(len(psi[s]), n ** 3, dtype=torch.complex128, device=DEVICE)
        grid[:, at] = psi[s]
        r = torch.fft.ifftn(grid.view(-1, n, n, n), dim=(1, 2, 3)).reshape(len(grid), -1) * n ** 3
        rho += (w[s, None] * (r.real ** 2 + r.imag ** 2)).sum(0)
    return rho


def exact(case, seed):
    c, n = case, case["grid"]
    if c["kind"] == "solve" and (c["iterations"] or c["atoms"] > 9):
        return None  # an unfinished iteration has no value of its own
    x = _inputs(c, seed)
    psi = x["psi"].to(torch.complex128)
    if c["kind"] == "hpsi":
        return _apply(x, n, psi)
    if c["kind"] == "overlap":
        return psi + _nonlocal(x["beta"], x["q"], psi)
    if c["kind"] == "density":
        return _density(x, n, psi)
    if c["kind"] == "gamma":  # the half-sphere vectors stand for real functions
        mil, ke = np.concatenate([x["mil"], -x["mil"][1:]]), np.concatenate([x["ke"], x["ke"][1:]])

        def whole(v):
            return torch.cat([v, v[:, 1:].conj()], dim=1)

        return _apply(x, n, whole(psi), mil, ke, whole(x["beta"]))[:, :len(x["ke"])].contiguous()
    npw = len(x["ke"])
    H = _apply(x, n, torch.eye(npw, dtype=torch.complex128, device=DEVICE)).T
    w, z = torch.linalg.eigh(0.5 * (H + H.conj().T))
    return {"eigenvalues": w[:c["bands"]], "density": _density(x, n, z[:, :c["bands"]].T.contiguous())}
