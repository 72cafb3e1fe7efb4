"""The calls whose speed matters to a user of this framework, as measurable cases.

Every case goes through the Python mirror of the C ABI (phoebe_b200.core), as the
tests and the benchmark do.  Inputs (force constants, band structures, couplings)
are made here from the seed: the cells, the spring models and the generators are
those of phoebe_b200.synth; the spring constants, the strength of every third-order
cell pair and the el-ph couplings change with the seed.  Band structures are
diagonalised here and handed to the framework as arrays, so that a builder case
does not depend on the band-structure kernels.

exact() restates each path in 64 bits with plain torch and numpy operations.
"""
import functools
import math

import numpy as np
import torch

from phoebe_b200 import constants as C
from phoebe_b200 import core, lattice, synth

TEMPS_K = (100.0, 300.0, 600.0)
ELPH_WINDOW = 0.3 / C.energyRyToEv
SIGMA_PH = 0.3 / C.ryToTHz
SIGMA_EL = 0.01


# ---------------------------------------------------------------------------
# cases
# ---------------------------------------------------------------------------

def _ph(name, cell, mesh, pairs, precision, smearing, temps, window=False, q2=0, iso=False, kind="linewidths"):
    return {"name": name, "kind": kind, "cell": cell, "n0": mesh[0], "n1": mesh[1], "n2": mesh[2],
            "pairs": pairs, "precision": precision, "smearing": smearing, "temps": temps,
            "window": window, "q2": q2, "iso": iso}


def _elph(name, ncell, n, factor, k1, precision, temps):
    return {"name": name, "kind": "elph", "ncell": ncell, "n": n, "factor": factor, "k1": k1,
            "precision": precision, "temps": temps}


def listed():
    return [
        # a convergence test's coarse mesh: everything is launches, copies and latency
        _ph("ph_split_5", "diamond", (5, 5, 5), 400, "split_fp16", "adaptive", 3),
        # the plain FP64 workload of the reference's size: 8^3, Gaussian 0.3 THz, 300 K
        _ph("ph_fp64_gauss_8", "diamond", (8, 8, 8), 400, "fp64", "gaussian", 1),
        # the headline: 20^3 linewidths in split precision, three temperatures
        _ph("ph_split_20", "diamond", (20, 20, 20), 400, "split_fp16", "adaptive", 3),
        # the plain FP64 path on a production mesh, with isotope and boundary scattering
        _ph("ph_fp64_16", "diamond", (16, 16, 16), 400, "fp64", "adaptive", 3, iso=True),
        # exact BTE solvers: the matrix is built in device memory (BF16 split, an odd
        # mesh, Gaussian) and multiplied with a few vectors
        _ph("matrix_bf16_odd", "diamond", (15, 13, 11), 400, "split_bf16", "gaussian", 1, kind="matrix"),
        # 15 branches, per-q1 windows, one rank's slice of q2, FP64
        _ph("perovskite_fp64", "perovskite", (24, 24, 24), 1500, "fp64", "adaptive", 1, window=True, q2=32),
        # the same in split precision
        _ph("perovskite_split", "perovskite", (24, 24, 24), 1500, "split_fp16", "adaptive", 1, window=True, q2=128),
        # 36 branches, one rank's slice of q2, split precision
        _ph("twelve_split", "twelve", (12, 12, 12), 400, "split_fp16", "adaptive", 1, q2=32),
        # carrier linewidths of a batch of outer k points, 343 x 343 vectors, split precision
        _elph("elph_split", 3, 20, 2, 64, "split_bf16", 1),
        # the same in FP64, a smaller batch
        _elph("elph_fp64", 3, 20, 2, 24, "fp64", 1),
        # the drop-in getCouplingsSquared of one q2 and a batch of q1, FP64
        {"name": "couplings_fp64", "kind": "couplings", "cell": "diamond", "pairs": 400, "q1": 1024,
         "precision": "fp64"},
        # the band structure of a mesh: 15 branches, 24^3 points, 7^3 force-constant grid
        {"name": "bands_perovskite_24", "kind": "bands", "cell": "perovskite", "n0": 24, "n1": 24, "n2": 24},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _mesh(rng, lo, hi):
    n = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return [max(2, int(round(n * rng.uniform(0.85, 1.15)))) for _ in range(3)]


def draw(rng):
    kind = rng.choice(["linewidths", "linewidths", "linewidths", "linewidths", "matrix", "elph", "elph",
                       "couplings", "bands"])
    precision = rng.choice(["fp64", "split_fp16", "split_bf16"])
    smearing = rng.choice(["adaptive", "gaussian"])
    if kind == "linewidths":
        cell = rng.choice(["diamond", "diamond", "perovskite", "twelve"])
        if cell == "diamond":
            mesh = _mesh(rng, 4, 13 if precision == "fp64" else 17)
            c = _ph("", cell, mesh, rng.choice([100, 250, 400]), precision, smearing, rng.randint(1, 3),
                    iso=rng.random() < 0.3)
        elif cell == "perovskite":
            mesh = _mesh(rng, 4, 20)
            nq = mesh[0] * mesh[1] * mesh[2]
            q2 = min(nq, _log_int(rng, 8, max(8, min(400, (300000 if precision == "fp64" else 900000) // nq))))
            c = _ph("", cell, mesh, rng.choice([300, 700, 1500]), precision, smearing, rng.randint(1, 3),
                    window=rng.random() < 0.6, q2=q2)
        else:
            mesh = _mesh(rng, 3, 10)
            nq = mesh[0] * mesh[1] * mesh[2]
            q2 = min(nq, _log_int(rng, 4, max(4, min(200, (12000 if precision == "fp64" else 50000) // nq))))
            c = _ph("", cell, mesh, 150, precision, smearing, rng.randint(1, 2), q2=q2)
    elif kind == "matrix":
        c = _ph("", "diamond", _mesh(rng, 4, 12), 400, precision, smearing, 1, kind="matrix")
    elif kind == "elph":
        c = _elph("", rng.choice([1, 2, 3]), _log_int(rng, 4, 20), rng.choice([1, 2]), _log_int(rng, 1, 64),
                  rng.choice(["fp64", "split_bf16"]), rng.randint(1, 2))
    elif kind == "couplings":
        c = {"kind": kind, "cell": rng.choice(["diamond", "diamond", "perovskite"]), "pairs": 300,
             "q1": _log_int(rng, 1, 2000), "precision": precision}
    else:
        cell = rng.choice(["diamond", "perovskite", "perovskite", "twelve"])
        m = _mesh(rng, 3, {"diamond": 28, "perovskite": 20, "twelve": 8}[cell])
        c = {"kind": kind, "cell": cell, "n0": m[0], "n1": m[1], "n2": m[2]}
    c.pop("name", None)
    return c


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------

def _rng(seed, tag):
    return np.random.default_rng([int(seed) & 0x7FFFFFFF, tag])


def _crystal(cell):
    return {"diamond": synth.diamond_crystal, "perovskite": synth.perovskite_crystal,
            "twelve": lambda: synth.twelve_atom_crystal(synth.SEED_BASE + 4)}[cell]()


@functools.lru_cache(maxsize=None)
def _fc2_base(cell):
    cr = _crystal(cell)
    if cell == "diamond":
        a = np.linalg.norm(cr.direct_cell[:, 0]) * np.sqrt(2.0)
        parts = [(a * np.sqrt(3.0) / 4.0, 45.0), (a / np.sqrt(2.0), 5.0)]
        grid = (4, 4, 4)
    elif cell == "perovskite":
        a = cr.direct_cell[0, 0]
        parts = [(0.5 * a, 12.0), (a / np.sqrt(2.0), 3.0), (a * np.sqrt(3.0) / 2.0, 2.0), (a, 1.5)]
        grid = (7, 7, 7)
    else:
        a = cr.direct_cell[0, 0]
        parts = [(a * np.sqrt(3.0) / 4.0, 40.0), (0.5 * a, 12.0), (a / np.sqrt(2.0), 5.0)]
        grid = (2, 2, 2)
    return [synth.spring_fc2(cr, [(r, synth._k_ry(k), None)], grid) for r, k in parts]


def _fc2(cell, seed):
    """Force constants of the cell's spring shells, each stiffness changed by up to 5%."""
    f = _rng(seed, 2).uniform(0.95, 1.05, 8)
    return sum(f[i] * p for i, p in enumerate(_fc2_base(cell)))


@functools.lru_cache(maxsize=4)
def _fc3_base(cell, pairs):
    return synth.random_fc3(_crystal(cell), pairs, synth.SEED_BASE, tol=1e-2, max_iter=6)


def _fc3(cell, pairs, seed):
    """The cell's third-order tensor, every cell pair's block changed by up to 20%."""
    b = _fc3_base(cell, pairs)
    f = _rng(seed, 3).uniform(0.8, 1.2, b.D3.shape[3:])
    return synth.FC3(b.D3 * f, b.R2, b.R3, b.w2, b.w3, b.num_pairs)


def _eigh(H, block=16384):
    """Batched Hermitian eigensolve (ascending); on the CPU beyond the GPU solver's batched size."""
    if H.shape[-1] > 32:
        E, V = np.linalg.eigh(H.cpu().numpy())
        return torch.from_numpy(E).to(H.device), torch.from_numpy(V).to(H.device)
    out = [torch.linalg.eigh(h) for h in H.split(block)]
    return torch.cat([o[0] for o in out]), torch.cat([o[1] for o in out])


def _bands(cell, fc2, q):
    """(E, U / sqrt(m), v) at Cartesian wavevectors q, from D(q) and its derivative."""
    cr = _crystal(cell)
    R, w, M = core.ws_reorder(cr, fc2)
    nb = cr.num_bands
    m = np.repeat(cr.atomic_masses, 3)
    dev = "cuda"
    Mw = torch.from_numpy((M * w[:, None, None] / np.sqrt(np.outer(m, m))).reshape(len(w), nb * nb)).to(dev)
    Rt = torch.from_numpy(R).to(dev)
    nz = Mw.abs().amax(1) > 0
    Mw, Rt = Mw[nz].to(torch.complex128), Rt[nz]
    E, U, V = [], [], []
    for qq in torch.from_numpy(q).to(dev).split(4096):
        ph = torch.exp(-1j * (qq @ Rt.T))
        D = (ph @ Mw).reshape(-1, nb, nb)
        w2, e = _eigh(0.5 * (D + D.conj().transpose(1, 2)))
        en = torch.sign(w2) * w2.abs().sqrt()
        v = torch.empty(len(qq), nb, 3, dtype=torch.float64, device=dev)
        for i in range(3):
            dD = ((-1j * Rt[:, i] * ph) @ Mw).reshape(-1, nb, nb)
            dD = 0.5 * (dD + dD.conj().transpose(1, 2))
            v[..., i] = (e.conj() * (dD @ e)).sum(1).real
        soft = en < 10 * C.phExcludeCutoff
        v = torch.where(soft[..., None], torch.zeros_like(v), v / (2 * torch.where(soft, torch.ones_like(en), en))[..., None])
        E.append(en)
        U.append(e / torch.from_numpy(np.sqrt(m)).to(dev)[:, None])
        V.append(v)
    return tuple(torch.cat(x).cpu().numpy() for x in (E, U, V))


def _neg_index(mesh):
    n0, n1, n2 = mesh
    i = np.arange(n0 * n1 * n2)
    return ((n2 - i // (n0 * n1)) % n2) * n0 * n1 + ((n1 - (i // n0) % n1) % n1) * n0 + (n0 - i % n0) % n0


def _mesh_bands(cell, mesh, seed):
    """Bands of a Gamma-centred mesh: one of q and -q diagonalised, the other its conjugate."""
    q = lattice.Mesh(_crystal(cell), mesh).cartesian_coords()
    neg = _neg_index(mesh)
    half = np.flatnonzero(np.arange(len(q)) <= neg)
    E, U, V = _bands(cell, _fc2(cell, seed), q[half])
    nb = E.shape[1]
    oE, oU, oV = np.empty((len(q), nb)), np.empty((len(q), nb, nb), np.complex128), np.empty((len(q), nb, 3))
    oE[neg[half]], oU[neg[half]], oV[neg[half]] = E, U.conj(), -V
    oE[half], oU[half], oV[half] = E, U, V
    oV[half[half == neg[half]]] = 0.0
    return oE, oU, oV


_kept = {}


def _context():
    """The one context that a program keeps."""
    if "ctx" not in _kept:
        _kept["ctx"] = core.Context(0)
    return _kept["ctx"]


def _ph_inputs(case, seed):
    cell, mesh = case["cell"], (case["n0"], case["n1"], case["n2"])
    E, U, V = _mesh_bands(cell, mesh, seed)
    nq = len(E)
    q2 = case["q2"] or nq
    return {"cell": cell, "mesh": mesh, "E": E, "U": U, "V": V, "fc3": _fc3(cell, case["pairs"], seed),
            "T": np.array([C.kelvin_to_ry(t) for t in TEMPS_K[:case["temps"]]]) if case["temps"] > 1
            else np.array([C.kelvin_to_ry(300.0)]),
            "window": synth.q2_window(E, mesh, synth.SEED_BASE + seed) if case["window"] else None,
            "iso": core.isotope_coupling(_crystal(cell), np.full(_crystal(cell).num_atoms, 2.0164e-4))
            if case["iso"] else None,
            "boundary": 1.0e6 if case["iso"] else 0.0,
            "q2b": (nq - q2) // 2, "q2e": (nq - q2) // 2 + q2,
            "x": _rng(seed, 5).normal(size=(3, 1, 3, nq * E.shape[1])) if case["kind"] == "matrix" else None}


def _el_inputs(case, seed):
    cr = synth.diamond_crystal()
    nw, nph, n = 8, 6, case["n"]
    kmesh, qmesh = (case["factor"] * n,) * 3, (n,) * 3
    Rh, degh, H = synth.wannier_hamiltonian(cr, nw, 3, synth.SEED_BASE + seed)
    Re, degE = synth.lattice_cube(cr, case["ncell"])
    k = lattice.Mesh(cr, kmesh).cartesian_coords()
    E, U, V = [], [], []
    Ht = torch.from_numpy(H.reshape(len(Rh), -1)).cuda()
    Rt = torch.from_numpy(Rh).cuda()
    for kk in torch.from_numpy(k).cuda().split(16384):
        ph = torch.exp(1j * (kk @ Rt.T))
        en, u = _eigh((ph @ Ht).reshape(-1, nw, nw))
        v = [(u.conj() * (((1j * Rt[:, i] * ph) @ Ht).reshape(-1, nw, nw) @ u)).sum(1).real for i in range(3)]
        E.append(en)
        U.append(u)
        V.append(torch.stack(v, -1))
    E, U, V = (torch.cat(x).cpu().numpy() for x in (E, U, V))
    Eq, Uq, _ = _mesh_bands("diamond", qmesh, seed)
    # couplings N(0,1) 0.1 eV/A exp(-(|Re|+|Rp|)/4 A), complex FP32
    d = torch.from_numpy(np.exp(-np.linalg.norm(Re, axis=1) * C.distanceBohrToAng / 4.0)).cuda()
    gen = torch.Generator(device="cuda").manual_seed(int(seed) * 7919 + 11)
    g = torch.randn(len(Re), len(Re), nph, nw, nw, 2, generator=gen, device="cuda")
    g *= (0.1 / C.energyRyToEv * C.distanceBohrToAng * d[:, None] * d).to(torch.float32)[:, :, None, None, None, None]
    g = torch.view_as_complex(g).cpu().numpy()
    mu = float(np.median(E))
    active = np.flatnonzero((np.abs(E - mu) <= ELPH_WINDOW).any(1))
    k1 = np.sort(_rng(seed, 7).choice(active, min(case["k1"], len(active)), replace=False)).astype(np.int32)
    T = np.array([C.kelvin_to_ry(t) for t in (300.0, 600.0)[:case["temps"]]])
    return {"cr": cr, "kmesh": kmesh, "qmesh": qmesh, "R": Re, "deg": degE, "g": g, "E": E, "U": U, "V": V,
            "Eq": Eq, "Uq": Uq, "mu": mu, "k1": k1, "T": T, "k": k}


def _coupling_inputs(case, seed):
    """One q2 and a batch of q1 of a generic mesh, with q3 = q1 +- q2."""
    cell = case["cell"]
    n, rng = case["q1"], _rng(seed, 4)
    B = _crystal(cell).reciprocal_cell
    q1, q2 = rng.uniform(0, 1, (n, 3)) @ B.T, rng.uniform(0, 1, 3) @ B.T
    _, U, _ = _bands(cell, _fc2(cell, seed), np.concatenate([q1, q1 + q2, q1 - q2, q2[None]]))
    return {"q1": q1, "q2": q2, "e1": U[:n], "e3p": U[n:2 * n], "e3m": U[2 * n:3 * n], "e2": U[-1],
            "fc3": _fc3(cell, case["pairs"], seed)}


def prepare(case, seed):
    ctx = _context()
    kind = case["kind"]
    if kind in ("linewidths", "matrix"):
        s = _ph_inputs(case, seed)
        cr = _crystal(s["cell"])
        bands = core.BandStructure.from_arrays(ctx, s["mesh"], cr.reciprocal_cell, s["E"], s["U"], s["V"])
        v3 = core.Interaction3Ph(ctx, cr, s["fc3"], precision=case["precision"])
        sm = core.PhScatteringMatrix(v3, bands, s["T"], case["smearing"], SIGMA_PH, window=s["window"],
                                     isotope_coupling=s["iso"], boundary_length=s["boundary"],
                                     in_memory=kind == "matrix")
        return {"kind": kind, "sm": sm, "q2": (s["q2b"], s["q2e"]), "whole": not case["q2"], "x": s["x"]}
    if kind == "elph":
        s = _el_inputs(case, seed)
        el = core.BandStructure.from_arrays(ctx, s["kmesh"], s["cr"].reciprocal_cell, s["E"], s["U"], s["V"])
        ph = core.BandStructure.from_arrays(ctx, s["qmesh"], s["cr"].reciprocal_cell, s["Eq"], s["Uq"])
        elph = core.InteractionElPhWan(ctx, s["R"], s["deg"], s["R"], s["deg"], s["g"])
        elph.setPrecision(case["precision"])
        sm = core.ElScatteringMatrix(elph, el, ph, s["T"], s["mu"], ELPH_WINDOW, "adaptive", SIGMA_EL)
        return {"kind": kind, "sm": sm, "k1": s["k1"]}
    if kind == "couplings":
        s = _coupling_inputs(case, seed)
        v3 = core.Interaction3Ph(ctx, _crystal(case["cell"]), s["fc3"], precision=case["precision"])
        return {"kind": kind, "v3": v3, **{k: s[k] for k in ("q1", "q2", "e1", "e2", "e3p", "e3m")}}
    h0 = core.PhononH0(ctx, _crystal(case["cell"]), _fc2(case["cell"], seed))
    return {"kind": kind, "h0": h0, "mesh": (case["n0"], case["n1"], case["n2"])}


def run(state):
    kind = state["kind"]
    if kind == "linewidths":
        b, e = state["q2"]
        return state["sm"].setup(b, e, finalize=state["whole"])
    if kind == "matrix":
        diag = state["sm"].setup()
        return [diag, state["sm"].offDiagonalDot(state["x"])]
    if kind == "elph":
        return state["sm"].setup(state["k1"])
    if kind == "couplings":
        v3 = state["v3"]
        v3.cacheD3(state["q2"])
        p, m = v3.getCouplingsSquared(state["q1"], state["q2"], state["e1"], state["e2"], state["e3p"], state["e3m"])
        return [np.stack(p), np.stack(m)]
    bands = state["h0"].populate(state["mesh"], withVelocities=True)
    E, U, v = bands.get()
    bands.close()
    return [E, U, v]


# ---------------------------------------------------------------------------
# work and tolerances
# ---------------------------------------------------------------------------

def _sizes(case):
    nb = {"diamond": 6, "perovskite": 15, "twelve": 36}[case["cell"]]
    return nb, case.get("n0", 0) * case.get("n1", 0) * case.get("n2", 0)


# distinct lattice vectors of the third-order pairs (the generator's own count)
_NR3 = {("diamond", 100): 19, ("diamond", 250): 39, ("diamond", 300): 41, ("diamond", 400): 43,
        ("perovskite", 300): 27, ("perovskite", 700): 57, ("perovskite", 1500): 67,
        ("twelve", 150): 19, ("twelve", 400): 33}


def work(case):
    kind = case["kind"]
    if kind == "elph":
        nv = (2 * case["ncell"] + 1) ** 3
        nk, nq, n1 = (case["factor"] * case["n"]) ** 3, case["n"] ** 3, case["k1"]
        x = 6 * 64
        bands = nk * (8 * 8 + 64 * 16 + 24 * 8) + nq * (6 * 8 + 36 * 16)
        # about three active bands on either side; half of the final states have one
        flops = n1 * (8 * nv * nv * x + 8 * nv * x * 3 + 0.5 * nq * (8 * nv * 6 * 3 * 8 + 8 * 6 * 6 * 3 * 8 + 8 * 6 * 3 * 3 * 8))
        return {"bytes": nv * nv * x * 8 + bands, "flops": flops}
    nb, nq = _sizes(case)
    if kind == "bands":
        # seven diagonalisations (the point and six displaced ones) of about 9 n^3 complex operations
        return {"bytes": nq * (nb * 8 + nb * nb * 16 + nb * 24), "flops": nq * 7 * 8 * 9 * nb ** 3}
    nr3 = _NR3[(case["cell"], case["pairs"])]
    fc3 = 8.0 * nb ** 3 * case["pairs"]
    if kind == "couplings":
        n = case["q1"]
        return {"bytes": fc3 + n * (3 * nb * nb * 16 + 24 + 2 * nb ** 3 * 8),
                "flops": 2 * n * (8 * nb ** 3 * nr3 + 24 * nb ** 4) + 8 * nb ** 3 * case["pairs"]}
    q2 = case["q2"] or nq
    vertices = q2 * nq * (0.6 if case["window"] else 1.0)
    nbytes = fc3 + nq * (nb * 8 + nb * nb * 16 + nb * 24) + 8 * case["temps"] * nq * nb
    if kind == "matrix":
        nbytes += 2 * 8.0 * (nq * nb) ** 2
    return {"bytes": nbytes, "flops": vertices * (8 * nb ** 3 * nr3 + 16 * nb ** 4)}


def tolerance(case):
    kind, p = case["kind"], case["precision"] if "precision" in case else "fp64"
    if kind == "bands":
        # energies agree to 3e-11; the group velocities are finite differences with a step of 1e-8
        return {"rel": 1e-6, "max": 1e-4}
    if p == "fp64":
        return {"rel": 1e-12, "max": 1e-11}
    if kind == "elph":
        # measured against 64 bits: 4.7e-6 and 6.6e-6
        return {"rel": 2e-5, "max": 4e-5}
    if kind == "matrix":
        # products without the diagonal cancel: 7.2e-6 and 2.0e-4 in BF16
        return {"rel": 1e-5, "max": 4e-4} if p == "split_fp16" else {"rel": 3e-5, "max": 8e-4}
    if kind == "couplings":
        # 5.7e-7 and 1.7e-6 in FP16, 3.5e-6 and 1.5e-5 in BF16
        return {"rel": 3e-6, "max": 1e-5} if p == "split_fp16" else {"rel": 1.5e-5, "max": 8e-5}
    # 1.0e-6 and 2.2e-6 in FP16, 2.5e-6 and 5.7e-6 in BF16
    return {"rel": 4e-6, "max": 1e-5} if p == "split_fp16" else {"rel": 1e-5, "max": 3e-5}


# ---------------------------------------------------------------------------
# the same results in plain 64-bit torch and numpy
# ---------------------------------------------------------------------------

def _deg_average(E, active=None):
    """(n, nb, nb) projection that averages over degenerate blocks (forward scan, 1e-6 Ry)."""
    n, nb = E.shape
    act = torch.ones_like(E, dtype=torch.bool) if active is None else active
    start = torch.zeros(n, nb, dtype=torch.int64, device=E.device)
    cur = torch.zeros(n, dtype=torch.int64, device=E.device)
    for b in range(nb):
        prev = act.gather(1, cur[:, None])[:, 0]
        same = ((E.gather(1, cur[:, None])[:, 0] - E[:, b]).abs() < C.degeneracyThreshold) & prev & act[:, b]
        cur = torch.where(same, cur, torch.full_like(cur, b))
        start[:, b] = cur
    S = (start[:, :, None] == start[:, None, :]).to(torch.float64)
    return S / S.sum(2, keepdim=True)


def _delta(smearing, e, sig):
    if smearing == "gaussian":
        x = e / sig
        return torch.where(x > 6.0, torch.zeros_like(x), torch.exp(-x * x) / (sig * C.sqrtPi))
    x = e / torch.where(sig == 0, torch.ones_like(sig), sig)
    d = torch.exp(-x * x) / (C.sqrtPi * C.erf2 * torch.where(sig == 0, torch.ones_like(sig), sig))
    d = torch.where((sig == 0) | (e.abs() > 2.0 * sig), torch.zeros_like(d), d)
    return torch.where((sig == 0) & (e == 0), torch.ones_like(d), d)   # no width and no mismatch: 1


def _width(P1, P2):
    """Adaptive width of two sets of projected velocities (.., 3), floored at 1e-4 eV."""
    s = ((P1 - P2).square().sum(-1) / 6.0).sqrt()
    return torch.where((s != 0) & (s < C.adaptiveBroadeningCutoff), torch.full_like(s, C.adaptiveBroadeningCutoff), s)


def _exact_ph(case, seed):
    s = _ph_inputs(case, seed)
    cr = _crystal(s["cell"])
    mesh, fc3, matrix = s["mesh"], s["fc3"], case["kind"] == "matrix"
    dev = "cuda"
    E, U, V = (torch.from_numpy(s[k]).to(dev) for k in "EUV")
    nq, nb = E.shape
    T = torch.from_numpy(s["T"]).to(dev)
    nT = len(T)
    n0, n1, n2 = mesh
    q = lattice.Mesh(cr, mesh).cartesian_coords()
    qt = torch.from_numpy(q).to(dev)
    neg = _neg_index(mesh)
    i = np.arange(nq)
    ix = torch.from_numpy(np.stack([i % n0, (i // n0) % n1, i // (n0 * n1)])).to(dev)
    nn = torch.tensor([n0, n1, n2], device=dev)[:, None]
    D3 = torch.from_numpy(np.ascontiguousarray(fc3.D3.transpose(4, 3, 0, 1, 2))).to(dev)   # r2 r3 a b c
    R2, R3 = torch.from_numpy(fc3.R2).to(dev), torch.from_numpy(fc3.R3).to(dev)
    nr2, nr3 = len(R2), len(R3)
    D3 = D3.reshape(nr2, -1)
    ph1 = torch.exp(-1j * (qt @ R3.T))                                    # q1, r3
    n = 1.0 / (torch.exp(E[None] / T[:, None, None]) - 1.0)
    n = torch.where(n < 0, torch.zeros_like(n), n)                        # T, q, b
    nt = n.permute(1, 2, 0).contiguous()                                  # q, b, T
    S = _deg_average(E)
    qT = torch.from_numpy(cr.reciprocal_cell / np.array(mesh)[:, None]).to(dev)
    P = V @ qT.T
    excl, low = E < C.phExcludeCutoff, E < C.phEnergyCutoff
    sigma = torch.tensor(SIGMA_PH, dtype=torch.float64, device=dev)
    out = torch.zeros(nT, nq, nb, dtype=torch.float64, device=dev)
    x = torch.from_numpy(s["x"]).to(dev).reshape(-1, nq, nb) if matrix else None
    y = torch.zeros_like(x) if matrix else None
    good1, inv = ~(excl | low), torch.where(low, torch.zeros_like(E), 1.0 / torch.where(low, torch.ones_like(E), E))
    win = None if s["window"] is None else [torch.from_numpy(w).to(dev) for w in s["window"]]
    norm = 1.0 / nq
    block = max(1, min(nq, int(6e7) // nb ** 3))
    for q2 in range(s["q2b"], s["q2e"]):
        m2 = int(neg[q2])
        ph2 = torch.exp(1j * (R2 @ qt[q2]))
        Y = torch.complex(ph2.real @ D3, ph2.imag @ D3).reshape(nr3, nb, nb, nb)
        Y = torch.einsum("ravc,vb->rabc", Y, U[q2])
        Dp = (torch.exp(-1j * (R3 @ qt[q2]))[:, None] * Y.reshape(nr3, -1))
        q3 = (ix + ix[:, q2:q2 + 1]) % nn
        q3 = q3[2] * n0 * n1 + q3[1] * n0 + q3[0]
        for b in range(0, nq, block):
            r = slice(b, min(nq, b + block))
            k3 = q3[r]
            t = (ph1[r] @ Dp).reshape(-1, nb, nb * nb)
            t = (U[r].transpose(1, 2) @ t).reshape(-1, nb * nb, nb)               # b1 b2, c
            t = t @ U[k3].conj()
            w = (t.real.square() + t.imag.square()).reshape(-1, nb, nb * nb)      # b1, b2 b3
            w = (S[r] @ w).reshape(-1, nb * nb, nb) @ S[k3]
            w = torch.matmul(S[q2], w.reshape(-1, nb, nb, nb))
            e1, e3 = E[r][:, :, None, None], E[k3][:, None, None, :]
            i3 = torch.where(E[k3] < C.phEnergyCutoff, torch.zeros_like(inv[k3]), inv[k3])
            for at, sign in ((q2, 1), (m2, -1)):
                if win is not None and not bool((win[0][at] <= win[1][r]).any()):
                    continue
                e2 = E[at][None, None, :, None]
                sg = sigma if case["smearing"] == "gaussian" else _width(P[at][None, :, None], P[k3][:, None])[:, None]
                pre = (good1[r] * inv[r])[:, :, None, None] * (good1[at] * inv[at])[:, None] * i3[:, None, None, :]
                pre = pre * w * (math.pi * 0.25 * norm)
                if win is not None:
                    pre = pre * (win[0][at] <= win[1][r])[:, None, None, None]
                if sign > 0:
                    d = pre * _delta(case["smearing"], e1 + e2 - e3, sg)
                else:
                    d1 = pre * _delta(case["smearing"], e1 + e3 - e2, sg)
                    d2 = pre * _delta(case["smearing"], e2 + e3 - e1, sg)
                b1, b2, b3 = nt[r][:, :, None], nt[at], nt[k3][:, None]                # .., T
                if sign > 0:
                    rate = (d @ (b3 + 1.0)) * b1 * b2
                else:
                    rate = (d1 @ b3) * b1 * (b2 + 1.0) + (d2 @ b3) * b2 * (b1 + 1.0)
                out[:, r] += 0.5 * rate.sum(2).permute(2, 0, 1)
                if matrix:
                    if b <= at < b + len(k3):
                        rate[at - b, :, :, 0].fill_diagonal_(0.0)
                    y[:, r] += sign * torch.einsum("qab,vb->vqa", rate[..., 0], x[:, at])
        if s["iso"] is not None:
            nat = nb // 3
            sg = sigma if case["smearing"] == "gaussian" else _width(P, torch.zeros_like(P))[:, :, None]
            d = _delta(case["smearing"], E[:, :, None] - E[q2], sg) * (1.0 if case["smearing"] == "gaussian" else 0.5)
            z = torch.einsum("qixa,ixb->qiab", U.conj().reshape(nq, nat, 3, nb), U[q2].reshape(nat, 3, nb))
            iso = torch.from_numpy(s["iso"]).to(dev)
            t = ((z.real.square() + z.imag.square()) * iso[:, None, None]).sum(1) * d * E[:, :, None] * E[q2]
            t = t * (math.pi * 0.5 * norm) * good1[:, :, None] * good1[q2]
            for c in range(nT):
                out[c] += (t * (n[c][:, :, None] * n[c, q2] + 0.5 * (n[c][:, :, None] + n[c, q2]))).sum(2)
    if not case["q2"]:
        if not matrix:
            A = ((E[:, :, None] - E[:, None, :]).abs() < C.degeneracyThreshold).to(torch.float64)
            out[0] = (A @ out[0][:, :, None]).squeeze(2) / A.sum(2)
        if s["boundary"] > 0:
            sh = torch.sinh(E[None] / 2.0 / T[:, None, None])
            out += torch.where(excl, torch.zeros_like(out), V.norm(dim=2) / s["boundary"] * 0.25 / sh / sh)
        out = torch.where(excl, torch.zeros_like(out), out)
    out = out.reshape(nT, -1).cpu().numpy()
    return [out, y.reshape(s["x"].shape).cpu().numpy()] if matrix else out


def _exact_elph(case, seed):
    s = _el_inputs(case, seed)
    dev = "cuda"
    E, U, V, Eq, Uq = (torch.from_numpy(s[k]).to(dev) for k in ("E", "U", "V", "Eq", "Uq"))
    kt, R = torch.from_numpy(s["k"]).to(dev), torch.from_numpy(s["R"]).to(dev)
    g = torch.from_numpy(s["g"]).to(dev).to(torch.complex128)
    nv, nph, nw, nq, n = len(R), 6, 8, len(Eq), case["n"]
    f, nk = case["factor"], case["factor"] * case["n"]
    T = torch.from_numpy(s["T"]).to(dev)
    i = torch.arange(nq, device=dev)
    iq = torch.stack([i % n, (i // n) % n, i // (n * n)]) * f
    qc = torch.from_numpy(lattice.Mesh(s["cr"], s["qmesh"]).cartesian_coords()).to(dev)
    php = torch.exp(1j * (qc @ R.T))
    P = V @ torch.from_numpy(s["cr"].reciprocal_cell / nk).to(dev).T
    act = (E >= s["mu"] - ELPH_WINDOW) & (E <= s["mu"] + ELPH_WINDOW)
    ok3 = Eq >= 5.0 / C.ryToCmm1
    i3 = torch.where(ok3, 1.0 / torch.where(ok3, Eq, torch.ones_like(Eq)), torch.zeros_like(Eq))
    S3 = _deg_average(Eq)
    out = torch.zeros(len(T), len(s["k1"]), nw, dtype=torch.float64, device=dev)
    for j, k1 in enumerate(s["k1"].tolist()):
        g1 = (torch.exp(1j * (R @ kt[k1])) @ g.reshape(nv, -1)).reshape(nv, nph, nw, nw)
        g1 = torch.einsum("rnvw,vb->rnbw", g1, U[k1])
        c = torch.tensor([k1 % nk, (k1 // nk) % nk, k1 // (nk * nk)], device=dev)[:, None]
        k2 = (iq + c) % nk
        k2 = k2[2] * nk * nk + k2[1] * nk + k2[0]
        g3 = (php @ g1.reshape(nv, -1)).reshape(nq, nph, nw * nw)
        g3 = (Uq.transpose(1, 2) @ g3).reshape(nq, nph * nw, nw) @ U[k2].conj()    # nu b1, b2
        w = (g3.real.square() + g3.imag.square()).reshape(nq, nph, nw, nw)
        a1, a2 = act[k1:k1 + 1], act[k2]
        w = (w * a1[0][:, None] * a2[:, None, None, :])
        w = _deg_average(E[k1:k1 + 1], a1)[0] @ w @ _deg_average(E[k2], a2)[:, None]
        w = (S3 @ w.reshape(nq, nph, nw * nw)).reshape(nq, nph, nw, nw)
        w = w * a1[0][:, None] * a2[:, None, None, :] * i3[:, :, None, None] * (math.pi / nq)
        de = (E[k1][None, :, None] - E[k2][:, None, :])[:, None]
        sg = _width(P[k1][None, :, None], P[k2][:, None])[:, None]
        w3 = Eq[:, :, None, None]
        d1, d2 = w * _delta("adaptive", de + w3, sg), w * _delta("adaptive", de - w3, sg)
        for t in range(len(T)):
            fe = 1.0 / (torch.exp((E[k2] - s["mu"]) / T[t]) + 1.0)[:, None, None, :]
            bo = (1.0 / (torch.exp(torch.where(ok3, Eq, torch.ones_like(Eq)) / T[t]) - 1.0))[:, :, None, None]
            out[t, j] = ((fe + bo) * d1 + (1.0 - fe + bo) * d2).sum((0, 1, 3))
        m = ((E[k1][:, None] - E[k1][None]).abs() < C.degeneracyThreshold) & a1[0][:, None] & a1[0][None]
        m = m.to(torch.float64)
        out[0, j] = (m @ out[0, j]) / m.sum(1).clamp(min=1.0)
    return out.cpu().numpy()


def _exact_couplings(case, seed):
    s = _coupling_inputs(case, seed)
    fc3 = s["fc3"]
    dev = "cuda"
    t = {k: torch.from_numpy(np.asarray(s[k])).to(dev) for k in ("q1", "q2", "e1", "e2", "e3p", "e3m")}
    R2, R3 = torch.from_numpy(fc3.R2).to(dev), torch.from_numpy(fc3.R3).to(dev)
    D3 = torch.from_numpy(np.ascontiguousarray(fc3.D3.transpose(4, 3, 0, 1, 2))).to(dev)
    nb, nr3 = D3.shape[2], D3.shape[1]
    ph1 = torch.exp(-1j * (t["q1"] @ R3.T))
    out = []
    for e3, conj in ((t["e3p"], False), (t["e3m"], True)):
        ph2, ph3 = torch.exp(1j * (R2 @ t["q2"])), torch.exp(-1j * (R3 @ t["q2"]))
        ph2, ph3, e2 = (ph2.conj(), ph3.conj(), t["e2"].conj()) if conj else (ph2, ph3, t["e2"])
        D = D3.reshape(len(R2), -1)
        Y = torch.complex(ph2.real @ D, ph2.imag @ D).reshape(nr3, nb, nb, nb) * ph3[:, None, None, None]
        Y = torch.einsum("ravc,vb->rabc", Y, e2)
        X = (ph1 @ Y.reshape(nr3, -1)).reshape(-1, nb, nb * nb)
        X = (t["e1"].transpose(1, 2) @ X).reshape(-1, nb * nb, nb) @ e3.conj()
        out.append((X.real.square() + X.imag.square()).reshape(-1, nb, nb, nb).cpu().numpy())
    return out


def _exact_bands(case, seed):
    """Energies only: eigenvectors have a phase of their own, velocities are finite differences."""
    q = lattice.Mesh(_crystal(case["cell"]), (case["n0"], case["n1"], case["n2"])).cartesian_coords()
    return [_bands(case["cell"], _fc2(case["cell"], seed), q)[0], None, None]


def exact(case, seed):
    kind = case["kind"]
    if kind in ("linewidths", "matrix"):
        return _exact_ph(case, seed)
    if kind == "elph":
        return _exact_elph(case, seed)
    if kind == "couplings":
        return _exact_couplings(case, seed)
    return _exact_bands(case, seed)
