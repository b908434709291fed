"""Timed cases of the band-solve path: the calls that a plane-wave program makes, through the public
entry points, over the sizes it meets.

The inputs are silicon-like cells built here from a seed: a local Gaussian pseudopotential and one s and
one p projector per atom, atoms near diamond sites (or anywhere in cells that are no multiple of the
diamond cell). A case gives the cell edges (A), the cutoff (Ry), the FFT box, the k-points, the bands:

* ``apply``     ``BatchedHamiltonian``: H c in float64, on a complex64 draft block, or in float32
                arithmetic on a complex128 block (the expansion applies of the mixed solver);
* ``gamma``     ``GammaHamiltonian.apply_phi``: the Gamma-point apply on real embedded rows;
* ``overlap``   ``BatchedHS.hs``: H c and S c of the generalized problem from one pass;
* ``density``   ``density_b``: rho(r) of a band block;
* ``precond``   ``torch.ops.gwb.precond_apply``: preconditioned residuals (learned network, or TPA);
* ``solve``     ``davidson_batched`` from the identity start, then the density of the solved bands;
* ``gsolve``    ``davidson_gamma`` (learned preconditioner, mixed precision), then the density.

The solves return eigenvalues and the density with Fermi occupations: eigenvectors are only defined up to
a phase (and a rotation inside a degenerate level), these are not.
"""

from __future__ import annotations

import math

import numpy as np
import torch

# one silicon-like species (local Gaussian, s and p Kleinman-Bylander channels), eV and A
HBAR2_2M = 13.605693122994 * 0.529177210903 ** 2
RY = 13.605693122994
LOC_A, LOC_SIGMA, PROJ_RC, PROJ_D = -23.2440, 0.42007, 0.65590, (-0.82907, 0.20251)
EDGE = 5.43            # cubic diamond cell
ATOM_VOLUME = 20.0     # A^3 per atom
SMEAR = 0.05           # eV, width of the Fermi occupations of the solved bands
SOLVE_TOL = 1e-10      # eV, the residual the solves run to

_DIAMOND = np.array([[0, 0, 0], [0, .5, .5], [.5, 0, .5], [.5, .5, 0],
                     [.25, .25, .25], [.25, .75, .75], [.75, .25, .75], [.75, .75, .25]])


def _case(kind, a, ecut, box, nk, nb, **more):
    a = (a, a, a) if isinstance(a, float) else a
    box = (box, box, box) if isinstance(box, int) else box
    return dict(kind=kind, cell=more.pop("cell", "box"), a0=a[0], a1=a[1], a2=a[2], ecut=ecut, n0=box[0], n1=box[1],
                n2=box[2], nk=nk, nb=nb, **more)


def listed():
    named = {
        # the smallest call: a primitive cell at Gamma in the box its cutoff asks for; launches and latency
        "apply_2_atoms": _case("apply", EDGE, 30.0, 25, 1, 8, cell="fcc", prec="f64"),
        # the complex64 draft of the two-stage solver: 8 atoms, 10 irreducible k, the cutoff's own box
        "apply_8_atoms_draft": _case("apply", EDGE, 40.0, 42, 10, 24, prec="c64"),
        # an elongated cell (layers, surfaces): unequal axes, odd band count
        "apply_24_atoms_layers": _case("apply", (EDGE, EDGE, 3 * EDGE), 30.0, (36, 36, 108), 4, 61, prec="f64"),
        # expansion apply of the mixed solver: 64 atoms, 4 k, 160 bands, pinned box
        "apply_64_atoms_expand": _case("apply", 2 * EDGE, 40.0, 72, 4, 160, prec="f32"),
        # float64 apply of a solve's certification, 64 atoms in the cutoff's own box, odd band count
        "apply_64_atoms": _case("apply", 2 * EDGE, 40.0, 84, 2, 129, prec="f64"),
        # the Gamma-only supercell: the whole block in float64 (polish, certification) ...
        "gamma_216_atoms": _case("gamma", 3 * EDGE, 30.0, 96, 1, 480, prec="f64"),
        # ... and expansion rows in float32 arithmetic, in the box its cutoff asks for
        "gamma_216_atoms_expand": _case("gamma", 3 * EDGE, 30.0, 108, 1, 331, prec="f32"),
        # density of a solved block, once per self-consistency step
        "density_64_atoms": _case("density", 2 * EDGE, 40.0, 72, 4, 160),
        # generalized (USPP/PAW) apply, H c and S c
        "overlap_8_atoms": _case("overlap", EDGE, 40.0, 36, 10, 24, prec="f64"),
        # learned preconditioner on the unconverged bands of a solve's round
        "precond_64_atoms": _case("precond", 2 * EDGE, 40.0, 72, 4, 160, n_add=101, net=True),
        # a whole solve of a small cell (float64, the default form) and its density
        "solve_8_atoms": _case("solve", EDGE, 40.0, 36, 10, 24),
        # a whole Gamma-only solve in the fast form, and its density: the largest work a user has
        "solve_216_atoms": _case("gsolve", 3 * EDGE, 30.0, 96, 1, 480),
    }
    return [dict(c, name=n) for n, c in named.items()]


def _good(n):
    while True:
        r = n
        for p in (2, 3, 5, 7):
            while r % p == 0:
                r //= p
        if r == 1:
            return n
        n += 1


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """Cells from 2 to about 200 atoms with equal or unequal edges, boxes that just hold the sphere or its
    products, 1 to 10 k, 1 to 480 bands."""
    kind = rng.choice(["apply"] * 6 + ["gamma"] * 3 + ["overlap"] * 2 + ["density"] * 2 + ["precond"] * 3 + ["solve"] * 2)
    if kind == "solve":
        ecut = round(rng.uniform(20.0, 40.0), 1)
        g = math.sqrt(ecut * RY / HBAR2_2M)
        m = int(g * EDGE / (2 * math.pi) + 0.87) + 1
        box = _good(rng.choice([2 * m + 1, 3 * m + 1]))
        return _case("solve", EDGE, ecut, box, rng.randint(1, 4), rng.randint(18, 28))
    while True:
        ecut = round(rng.uniform(20.0, 40.0), 1)
        a = [round(math.exp(rng.uniform(math.log(4.2), math.log(16.3))), 2) for _ in range(3)]
        if rng.random() < 0.5:
            a = [a[0]] * 3
        vol = a[0] * a[1] * a[2]
        g = math.sqrt(ecut * RY / HBAR2_2M)
        # the sphere's reach per axis (any k), then a box that holds it, 3/2 or twice its width
        wide = rng.choice([2.0, 3.0, 4.0])
        box = [_good(int(wide * (g * x / (2 * math.pi) + 0.87)) + 2) for x in a]
        n = box[0] * box[1] * box[2]
        nk = 1 if kind == "gamma" else _log_int(rng, 1, 10)
        nb = _log_int(rng, 1, 480 if kind == "gamma" else 200)
        atoms = max(1, round(vol / ATOM_VOLUME))
        if max(box) <= 112 and vol <= 4400 and nk * atoms <= 260 and nk * nb * n <= 3.0e8:
            break
    more = {}
    if kind in ("apply", "overlap"):
        more["prec"] = rng.choice(["f64", "f64", "c64", "f32"] if kind == "apply" else ["f64", "c64"])
    if kind == "gamma":
        more["prec"] = rng.choice(["f64", "f32"])
    if kind == "precond":
        more["n_add"], more["net"] = rng.randint(1, nb), rng.random() < 0.6
    return _case(kind, tuple(a), ecut, tuple(box), nk, nb, **more)


# ---------------------------------------------------------------------------
# the cell of a case


def _shape(case):
    return case["n0"], case["n1"], case["n2"]


def _cell(case):
    a = np.array([case["a0"], case["a1"], case["a2"]])
    if case["cell"] == "fcc":
        return 0.5 * a[:, None] * np.array([[0.0, 1, 1], [1, 0, 1], [1, 1, 0]])
    return np.diag(a)


def _atoms(case):
    return 2 if case["cell"] == "fcc" else max(1, round(case["a0"] * case["a1"] * case["a2"] / ATOM_VOLUME))


def _positions(case, gen):
    """Fractional positions: diamond sites displaced by 0.05 A where the cell is a multiple of the diamond
    cell, else anywhere."""
    cell = _cell(case)
    reps = [case[k] / EDGE for k in ("a0", "a1", "a2")]
    if case["cell"] == "fcc":
        base = np.array([[0.0, 0, 0], [0.25, 0.25, 0.25]])
    elif all(abs(r - round(r)) < 1e-6 for r in reps):
        s = np.stack(np.meshgrid(*[np.arange(round(r)) for r in reps], indexing="ij"), -1).reshape(-1, 1, 3)
        base = ((s + _DIAMOND) / np.array([round(r) for r in reps])).reshape(-1, 3)
    else:
        return gen.random((_atoms(case), 3))
    return base + gen.normal(0.0, 0.05, base.shape) @ np.linalg.inv(cell)


def _kpoints(nk):
    ks = [(i / 4, j / 4, l / 4) for i in range(3) for j in range(i + 1) for l in range(j + 1)]
    return np.array(ks[:nk])


def _spheres(case):
    """Per k: Miller indices, k+G, |k+G|^2 and box index of |k+G|^2 below the cutoff, by length."""
    cell, ecut = _cell(case), case["ecut"] * RY
    b = 2 * np.pi * np.linalg.inv(cell).T
    g = math.sqrt(ecut / HBAR2_2M)
    reach = [int(g * np.linalg.norm(cell[i]) / (2 * np.pi) + 1) + 1 for i in range(3)]
    cand = np.stack(np.meshgrid(*[np.arange(-r, r + 1) for r in reach], indexing="ij"), -1).reshape(-1, 3)
    n0, n1, n2 = _shape(case)
    out = []
    for k in _kpoints(case["nk"]):
        kpg = (cand + k) @ b
        q2 = (kpg * kpg).sum(1)
        on = HBAR2_2M * q2 <= ecut
        m, kpg, q2 = cand[on], kpg[on], q2[on]
        o = np.lexsort((m[:, 2], m[:, 1], m[:, 0], np.round(q2, 9)))
        m, kpg, q2 = m[o], kpg[o], q2[o]
        out.append((k, m, kpg, q2, (m[:, 0] % n0) * n1 * n2 + (m[:, 1] % n1) * n2 + m[:, 2] % n2))
    return out


def _potential(case, frac, dev):
    cell = _cell(case)
    b = 2 * np.pi * np.linalg.inv(cell).T
    n = _shape(case)
    m = [torch.fft.fftfreq(k, d=1.0 / k, dtype=torch.float64, device=dev) for k in n]
    ph = [torch.exp(-2j * math.pi * torch.as_tensor(frac[:, i], device=dev)[:, None] * m[i]) for i in range(3)]
    s = ((ph[0][:, :, None] * ph[1][:, None, :]).reshape(len(frac), -1).T @ ph[2]).reshape(n)
    grid = torch.stack(torch.meshgrid(*m, indexing="ij"), -1) @ torch.as_tensor(b, device=dev)
    v = s * (LOC_A / abs(np.linalg.det(cell)) * torch.exp(-0.5 * LOC_SIGMA ** 2 * (grid * grid).sum(-1)))
    return (torch.fft.ifftn(v) * (n[0] * n[1] * n[2])).real.contiguous()


def _projectors(kpg, tau, vol):
    """(4 atoms, npw): per atom its s and p columns."""
    q2 = (kpg * kpg).sum(1)
    f = torch.exp(-0.5 * PROJ_RC ** 2 * q2)
    c = 4 * math.pi / math.sqrt(vol)
    s = (c * 0.5 / math.sqrt(math.pi) * f).to(torch.complex128)
    p = -1j * c * math.sqrt(3 / (4 * math.pi)) * PROJ_RC * f * kpg.T[[2, 0, 1]]
    cols = torch.cat([s[None], p])                                           # (4, npw)
    phase = torch.exp(-1j * (tau @ kpg.T))                                   # (atoms, npw)
    return (phase[:, None, :] * cols[None]).reshape(-1, kpg.shape[0])


def _system(case, seed):
    """The tables of a case: everything below is plain numpy and torch on the GPU."""
    dev = torch.device("cuda", torch.cuda.current_device())
    rng = np.random.default_rng(seed)
    cell = _cell(case)
    vol = abs(np.linalg.det(cell))
    frac = _positions(case, rng)
    tau = torch.as_tensor(frac @ cell, device=dev)
    sph = _spheres(case)
    nk, npw = len(sph), max(len(s[3]) for s in sph)
    t = np.zeros((nk, npw))
    flat = np.zeros((nk, npw), dtype=np.int64)
    mask = np.zeros((nk, npw), dtype=bool)
    kpg = np.zeros((nk, npw, 3))
    p = torch.zeros(nk, 4 * len(frac), npw, dtype=torch.complex128, device=dev)
    for i, (_, _, kg, q2, fl) in enumerate(sph):
        n = len(q2)
        t[i, :n], flat[i, :n], mask[i, :n], kpg[i, :n] = HBAR2_2M * q2, fl, True, kg
        p[i, :, :n] = _projectors(torch.as_tensor(kg, device=dev), tau, vol)
    dij = torch.diag(torch.tensor([PROJ_D[0]] + 3 * [PROJ_D[1]], dtype=torch.float64, device=dev).repeat(len(frac)))
    gen = torch.Generator(device=dev).manual_seed(int(seed))
    return dict(dev=dev, sph=sph, vol=vol, t=torch.as_tensor(t, device=dev), flat=torch.as_tensor(flat, device=dev),
                mask=torch.as_tensor(mask, device=dev), kpg=torch.as_tensor(kpg, device=dev), p=p, dij=dij,
                v=_potential(case, frac, dev), gen=gen, npw=[len(s[3]) for s in sph], atoms=len(frac))


def _batched(s):
    from gradwave_b200.basis import BatchedK
    dev = s["dev"]
    return BatchedK(torch.tensor(s["npw"], device=dev), s["mask"], s["flat"], s["kpg"], s["t"],
                    torch.zeros(0, dtype=torch.complex128, device=dev),
                    torch.arange(s["atoms"], device=dev).repeat_interleave(4), s["dij"])


def _rows(s, nk, nb, npw):
    """Unit rows whose amplitude falls with the kinetic energy, as bands do."""
    c = torch.randn(nk, nb, npw, 2, dtype=torch.float64, device=s["dev"], generator=s["gen"])
    c = torch.view_as_complex(c) * (s["mask"] / (1.0 + s["t"] / 10.0) ** 2)[:, None, :]
    return c / torch.linalg.vector_norm(c, dim=-1, keepdim=True)


def _gamma_basis(case, s):
    from gradwave_b200.basis import GSphere
    from gradwave_b200.gamma import build_gamma_basis
    k, m, kpg, q2, flat = s["sph"][0]
    return build_gamma_basis(GSphere(k, m, kpg, q2, flat), _shape(case))


def _augmentation(s):
    """A small symmetric q per atom (overlap charges of the s and p channels)."""
    q = torch.randn(s["atoms"], 4, 4, dtype=torch.float64, device=s["dev"], generator=s["gen"])
    return torch.block_diag(*(0.02 * (q + q.transpose(1, 2))))


def _residual_state(case, s):
    """Ritz rows, residuals (largest at high kinetic energy), eigenvalues and the selected bands."""
    nk, nb, npw = case["nk"], case["nb"], s["t"].shape[1]
    x = _rows(s, nk, nb, npw)
    r = _rows(s, nk, nb, npw) * (1e-3 * (1.0 + s["t"] / 5.0))[:, None, :]
    eig = torch.sort(20.0 * torch.rand(nk, nb, dtype=torch.float64, device=s["dev"], generator=s["gen"]) - 5.0, dim=1)[0]
    sel = torch.argsort(torch.rand(nk, nb, device=s["dev"], generator=s["gen"]), dim=1)[:, : case["n_add"]]
    return x, r, eig, sel.to(torch.int32).contiguous()


def _fermi(eig, weights, electrons):
    """Fermi occupations of the sorted levels, the level set halfway between the last filled and the next."""
    e = torch.sort(eig.reshape(-1))[0]
    n = min(electrons // 2 * eig.shape[0], e.numel() - 1)
    mu = 0.5 * (e[n - 1] + e[n])
    return 2.0 * torch.sigmoid((mu - eig) / SMEAR)


def prepare(case, seed):
    from gradwave_b200 import _lib
    from gradwave_b200.gamma import GammaHamiltonian, gamma_start
    from gradwave_b200.hamiltonian import BatchedHamiltonian
    from gradwave_b200.learned import LearnedPreconditioner
    from gradwave_b200.uspp import BatchedHS
    s = _system(case, seed)
    kind, nk, nb, shape = case["kind"], case["nk"], case["nb"], _shape(case)
    npw = s["t"].shape[1]
    st = dict(case=case, shape=shape, vol=s["vol"], kw=torch.full((nk,), 1.0 / nk, dtype=torch.float64, device=s["dev"]))
    if kind in ("gamma", "gsolve"):
        gb = _gamma_basis(case, s)
        st["h"] = GammaHamiltonian(gb, s["v"], s["p"][0], s["dij"])
        if kind == "gamma":
            phi = torch.randn(nb, npw, dtype=torch.float64, device=s["dev"], generator=s["gen"])
            phi = phi / (1.0 + st["h"].t_phi / 10.0) ** 2
            st["phi"] = phi / torch.linalg.vector_norm(phi, dim=1, keepdim=True)
            st["prec"] = _lib.GWB_FP64 if case["prec"] == "f64" else _lib.GWB_FP32
        else:
            st.update(gb=gb, bk=_batched(s), x0=gamma_start(gb, nb, s["dev"]), electrons=4 * s["atoms"],
                      net=LearnedPreconditioner.load(device=s["dev"]))
        return st
    if kind == "precond":
        st["x"], st["r"], st["eig"], st["sel"] = _residual_state(case, s)
        st["t"] = s["t"]
        st["params"] = LearnedPreconditioner.load(device=s["dev"]).params if case["net"] else None
        return st
    bk = _batched(s)
    if kind == "density":
        st["c"], st["bk"] = _rows(s, nk, nb, npw), bk
        st["occ"] = 2.0 * torch.rand(nk, nb, dtype=torch.float64, device=s["dev"], generator=s["gen"])
        return st
    if kind == "overlap":
        st["h"] = BatchedHS(bk, shape, s["v"], s["p"], s["dij"], _augmentation(s))
    else:
        st["h"] = BatchedHamiltonian(bk, shape, s["v"], s["p"])
    if kind == "solve":
        x0 = torch.zeros(nk, nb, npw, dtype=torch.complex128, device=s["dev"])
        x0[:, torch.arange(nb), torch.arange(nb)] = 1.0
        st.update(bk=bk, x0=x0, electrons=4 * s["atoms"])
    else:
        c = _rows(s, nk, nb, npw)
        st["c"] = c.to(torch.complex64) if case["prec"] == "c64" else c
    return st


def run(st):
    from gradwave_b200.davidson import davidson_batched
    from gradwave_b200.density import density_b
    from gradwave_b200.gamma import davidson_gamma, half_to_full
    case = st["case"]
    kind = case["kind"]
    if kind == "apply":
        return st["h"].apply_fp32(st["c"]) if case["prec"] == "f32" else st["h"].apply(st["c"])
    if kind == "gamma":
        return st["h"].apply_phi(st["phi"], prec=st["prec"])
    if kind == "overlap":
        return list(st["h"].hs(st["c"]))
    if kind == "density":
        return density_b(st["c"], st["occ"], st["kw"], st["bk"], st["shape"], st["vol"])
    if kind == "precond":
        return torch.ops.gwb.precond_apply(st["x"], st["r"], st["t"], st["sel"], st["eig"], st["params"], None)
    if kind == "solve":
        res = davidson_batched(st["h"].apply, st["x0"], st["bk"].t, st["bk"].mask, tol=SOLVE_TOL, max_iter=200)
        occ = _fermi(res.eigenvalues, st["kw"], st["electrons"])
        return [res.eigenvalues, st["h"].density(res.eigenvectors, occ, st["kw"], st["vol"])]
    res = davidson_gamma(st["h"], st["x0"], tol=SOLVE_TOL, max_iter=200, mode="mixed", n_buffer=16, precond=st["net"])
    occ = _fermi(res.eigenvalues[None], st["kw"], st["electrons"])
    full = half_to_full(st["gb"], res.eigenvectors)[None]
    return [res.eigenvalues, density_b(full, occ, st["kw"], st["bk"], st["shape"], st["vol"])]


# ---------------------------------------------------------------------------
# what a pass cannot do without


def work(case):
    kind, nk, nb = case["kind"], case["nk"], case["nb"]
    n = case["n0"] * case["n1"] * case["n2"]
    g = math.sqrt(case["ecut"] * RY / HBAR2_2M)
    vol = abs(np.linalg.det(_cell(case)))
    npw = vol * g ** 3 / (6 * math.pi ** 2)         # plane waves of one k
    nproj = 4 * _atoms(case)
    fft = 5.0 * n * math.log2(n)                    # one transform of one complex row
    prec = case.get("prec", "f64")
    es = 8 if prec == "c64" else 16                 # bytes of a coefficient
    ps = 16 if prec == "f64" else 8                 # bytes of a projector coefficient in the arithmetic used
    rows = nk * nb
    nl = 8.0 * nproj * npw                          # one complex product of a row with the projectors
    tables = nk * nproj * npw * ps + 8.0 * n + 8.0 * nk * npw
    if kind == "apply":
        return {"bytes": 2 * rows * npw * es + tables, "flops": rows * (2 * fft + 2 * nl)}
    if kind == "gamma":                             # two real rows to a transform, real products
        return {"bytes": 2 * rows * npw * 8 + tables / 2, "flops": rows * (fft + nl / 2)}
    if kind == "overlap":
        return {"bytes": 3 * rows * npw * es + tables, "flops": rows * (2 * fft + 3 * nl)}
    if kind == "density":
        return {"bytes": rows * npw * es + 8.0 * n, "flops": rows * (fft + 4.0 * n)}
    if kind == "precond":
        sel = nk * case["n_add"] * npw
        return {"bytes": 3 * 16.0 * sel + 8.0 * nk * npw, "flops": sel * (30.0 + (17000.0 if case["net"] else 0.0))}
    # A solve: bands, eigenvectors and tables once for the bytes; for the operations the applies and the
    # subspace products (four projections, two triangular transforms, two Ritz blocks, one column block) of
    # the rounds that such a solve cannot do without, about 20
    rounds = 20
    sub = 8.0 * npw * nb * 14 * nb
    if kind == "solve":
        return {"bytes": 2 * rows * npw * es + tables + 8.0 * n, "flops": rounds * (rows * (2 * fft + 2 * nl) + nk * sub)}
    return {"bytes": 2 * rows * npw * 8 + tables / 2 + 8.0 * n, "flops": rounds * (rows * (fft + nl / 2) + sub / 4)}


def tolerance(case):
    kind, prec = case["kind"], case.get("prec", "f64")
    if kind in ("solve", "gsolve"):
        # eigenvalues are second order in the residual (1e-10 eV), the density first order; start blocks
        # 1e-13 apart gave 1.6e-13 at most
        return {"rel": 1e-10, "max": 1e-8}
    if kind == "precond":
        # TPA is float64; the network has BF16 weights and activations
        return {"rel": 1.5e-2, "max": 0.3} if case["net"] else {"rel": 1e-12, "max": 1e-10}
    if prec == "f64":
        return {"rel": 5e-15, "max": 1e-12}
    # float32 transforms (1.4e-7 from 64 bits); from 128 projectors the float32 arithmetic of complex128
    # blocks contracts them in split BF16 (1.4e-6)
    return {"rel": 6e-7, "max": 6e-5} if prec == "c64" else {"rel": 5e-6, "max": 5e-4}


# ---------------------------------------------------------------------------
# the same results in 64 bits, by torch


def _local(s, shape, k, c, chunk=16):
    """Box product of the rows c of one k: scatter, inverse transform, v(r), transform, gather."""
    n = shape[0] * shape[1] * shape[2]
    np_k = s["npw"][k]
    idx = s["flat"][k, :np_k]
    out = torch.zeros_like(c)
    for b in range(0, c.shape[0], chunk):
        cb = c[b:b + chunk, :np_k]
        box = torch.zeros(cb.shape[0], n, dtype=torch.complex128, device=c.device)
        box[:, idx] = cb
        psi = torch.fft.ifftn(box.view(-1, *shape), dim=(1, 2, 3)) * s["v"]
        out[b:b + chunk, :np_k] = torch.fft.fftn(psi, dim=(1, 2, 3)).reshape(-1, n)[:, idx]
    return out


def _apply(s, shape, c, mat=None):
    """H c (and c + P^T q P* c with a second matrix)."""
    h, o = torch.empty_like(c), torch.empty_like(c)
    for k in range(c.shape[0]):
        b = c[k] @ s["p"][k].conj().T
        h[k] = s["t"][k] * c[k] + _local(s, shape, k, c[k]) + (b @ s["dij"].to(b.dtype)) @ s["p"][k]
        if mat is not None:
            o[k] = c[k] + (b @ mat.to(b.dtype)) @ s["p"][k]
    return h if mat is None else [h, o]


def _density(s, shape, c, occ, chunk=16):
    n = shape[0] * shape[1] * shape[2]
    rho = torch.zeros(shape, dtype=torch.float64, device=c.device)
    for k in range(c.shape[0]):
        np_k = s["npw"][k]
        for b in range(0, c.shape[1], chunk):
            cb = c[k, b:b + chunk, :np_k]
            box = torch.zeros(cb.shape[0], n, dtype=torch.complex128, device=c.device)
            box[:, s["flat"][k, :np_k]] = cb
            psi = torch.fft.ifftn(box.view(-1, *shape), dim=(1, 2, 3), norm="forward")
            rho += ((psi.real ** 2 + psi.imag ** 2) * occ[k, b:b + chunk, None, None, None]).sum(0)
    return rho / (c.shape[0] * s["vol"])


def _network(par, u):
    h = 64
    w1, b1, w2, b2, w3, b3, w4, b4 = torch.split(par, [4 * h, h, h * h, h, h * h, h, h, 1])
    z = torch.nn.functional.silu(u @ w1.view(h, 4).T + b1)
    z = torch.nn.functional.silu(z @ w2.view(h, h).T + b2)
    z = torch.nn.functional.silu(z @ w3.view(h, h).T + b3)
    return z @ w4 + b4


def _precond(s, x, r, eig, sel, par):
    out = torch.empty(*sel.shape, x.shape[2], dtype=torch.complex128, device=x.device)
    for k in range(x.shape[0]):
        for j, b in enumerate(sel[k].tolist()):
            t, xb, rb = s["t"][k], x[k, b], r[k, b]
            tb = (t * (xb.real ** 2 + xb.imag ** 2)).sum()
            y = t / tb
            num = 27 + 18 * y + 12 * y ** 2 + 8 * y ** 3
            f = num / (num + 16 * y ** 4)
            if par is not None:
                rabs = rb.abs()
                rms = torch.linalg.vector_norm(rb) / math.sqrt(rb.numel())
                u = torch.stack([torch.log1p(y), (eig[k, b] / tb).clamp(-8, 8).expand_as(y) / 4,
                                 torch.log10(rabs / rms + 1e-6) / 3,
                                 torch.log10(tb.clamp_min(1e-3) / 10).expand_as(y)], -1)
                f = f * torch.exp(_network(par, u).clamp(-3, 3))
            d = f * rb
            out[k, j] = d / torch.linalg.vector_norm(d)
    return out


def _dense_solve(case, s):
    """Lowest bands of the dense Hamiltonian of every k, and their density."""
    shape, nb = _shape(case), case["nb"]
    n = shape[0] * shape[1] * shape[2]
    eig, vec = [], torch.zeros(case["nk"], nb, s["t"].shape[1], dtype=torch.complex128, device=s["dev"])
    vg = torch.fft.fftn(s["v"].to(torch.complex128)).reshape(-1) / n
    for k, (_, m, _, _, _) in enumerate(s["sph"]):
        np_k = len(m)
        m = torch.as_tensor(m, device=s["dev"])
        d = [(m[:, None, i] - m[None, :, i]) % shape[i] for i in range(3)]
        p = s["p"][k, :, :np_k]
        h = vg[(d[0] * shape[1] + d[1]) * shape[2] + d[2]]
        h += p.T @ (s["dij"].to(p.dtype) @ p.conj())
        h.diagonal().add_(s["t"][k, :np_k])
        w, u = torch.linalg.eigh(h)
        eig.append(w[:nb])
        vec[k, :, :np_k] = u[:, :nb].T
    eig = torch.stack(eig)
    return [eig, _density(s, shape, vec, _fermi(eig, None, 4 * s["atoms"]))]


def exact(case, seed):
    kind, nk, nb, shape = case["kind"], case["nk"], case["nb"], _shape(case)
    if kind == "gsolve":
        return None
    s = _system(case, seed)
    npw = s["t"].shape[1]
    if kind == "solve":  # dense eigenvectors: seconds for each k of a few thousand plane waves
        return _dense_solve(case, s) if nk * npw ** 3 < 4.5 * 4600.0 ** 3 else None
    if kind == "gamma":
        return _exact_gamma(case, s)
    if kind == "precond":
        x, r, eig, sel = _residual_state(case, s)
        par = None
        if case["net"]:
            from gradwave_b200.learned import WEIGHTS
            par = torch.as_tensor(np.load(WEIGHTS), device=s["dev"]).double()
        return _precond(s, x, r, eig, sel, par)
    if kind == "overlap":
        q = _augmentation(s)
        c = _rows(s, nk, nb, npw)
        c = c.to(torch.complex64).to(torch.complex128) if case["prec"] == "c64" else c
        return _apply(s, shape, c, q)
    c = _rows(s, nk, nb, npw)
    if kind == "density":
        return _density(s, shape, c, 2.0 * torch.rand(nk, nb, dtype=torch.float64, device=s["dev"], generator=s["gen"]))
    return _apply(s, shape, c.to(torch.complex64).to(torch.complex128) if case["prec"] == "c64" else c)


def _exact_gamma(case, s):
    """The complex apply on the full sphere of the rows that the embedded rows stand for: slot 0 is G = 0,
    then (re, im) sqrt(2) of one G of each pair, the one positive in (m3, m2, m1)."""
    m = s["sph"][0][1]
    n = _shape(case)
    dev, npw = s["dev"], len(m)
    zero = np.all(m == 0, axis=1)
    pos = (m[:, 2] > 0) | ((m[:, 2] == 0) & ((m[:, 1] > 0) | ((m[:, 1] == 0) & (m[:, 0] > 0))))
    rep = np.concatenate([np.flatnonzero(zero), np.flatnonzero(pos)])
    where = np.full(n[0] * n[1] * n[2], -1, dtype=np.int64)

    def flat(a):
        return (a[:, 0] % n[0]) * n[1] * n[2] + (a[:, 1] % n[1]) * n[2] + a[:, 2] % n[2]

    where[flat(m)] = np.arange(npw)
    partner = torch.as_tensor(where[flat(-m[rep])], device=dev)
    rep = torch.as_tensor(rep, device=dev)
    t_phi = torch.repeat_interleave(s["t"][0, rep], 2)[1:]
    phi = torch.randn(case["nb"], npw, dtype=torch.float64, device=dev, generator=s["gen"])
    phi = phi / (1.0 + t_phi / 10.0) ** 2
    phi = phi / torch.linalg.vector_norm(phi, dim=1, keepdim=True)
    out = torch.empty_like(phi)
    for b in range(0, case["nb"], 64):
        half = torch.complex(phi[b:b + 64, 1::2], phi[b:b + 64, 2::2]) / math.sqrt(2.0)
        c = torch.zeros(1, half.shape[0], npw, dtype=torch.complex128, device=dev)
        c[0][:, rep[0]] = phi[b:b + 64, 0].to(torch.complex128)
        c[0][:, partner[1:]] = half.conj()
        c[0][:, rep[1:]] = half
        h = _apply(s, n, c)[0][:, rep]
        out[b:b + 64, 0] = h[:, 0].real
        out[b:b + 64, 1::2] = math.sqrt(2.0) * h[:, 1:].real
        out[b:b + 64, 2::2] = math.sqrt(2.0) * h[:, 1:].imag
    return out
