"""The split-precision kernel with one warp per q1 (cells of up to 36 branches) at the edges of its
classes of tile and of its lanes' tiles, against the FP64 builder on the same band structure: the
split paths' bar of 1e-5 on linewidths above 1e-8 of the largest.  Cells of 1 to 12 atoms (the
twelve-atom cell's first atoms), q1 counts that are no multiple of an item, R3 counts of one K step
and of several A stages, q2 windows, both smearings, and an R3 count that leaves no room for the
kernel (the older one takes over).  The FP64 builders of up to 16 branches against the oracle at the
1e-10 of the other FP64 linewidth tests: as routed, where problems as small as these run on the
shared-memory builder, and forced onto the many-branch one (FP64 tensor pipe, wide.cu's kernel up to 6
branches); the route between the two; isotope scattering in slots of q2."""
import numpy as np
import pytest

import oracle
from phoebe_b200 import constants as C
from phoebe_b200 import lattice, synth

pytestmark = pytest.mark.gpu


def _cell(nat):
    cr = synth.twelve_atom_crystal(synth.SEED_BASE + 4)
    return lattice.Crystal(cr.direct_cell, cr.positions[:nat], np.arange(nat), cr.species_masses[:nat])


def _fc3(cr, nr3):
    R, _ = synth.lattice_cube(cr, 3)
    rng = np.random.default_rng(nr3)
    o = np.argsort(np.linalg.norm(R, axis=1), kind="stable")
    nat, nb = cr.num_atoms, cr.num_bands
    D3 = rng.normal(size=(nb, nb, nb, nr3, 1)) * 0.05
    return synth.FC3(D3, R[o[1:2]], R[o[:nr3]], np.ones((1, nat, nat)), np.ones((nr3, nat, nat)), nr3)


def _bands(ctx, cr, mesh, rng):
    """Energies with degenerate blocks in every point, random unitary eigenvectors; -q the conjugate of q."""
    from phoebe_b200.core import BandStructure
    n0, n1, n2 = mesh
    nq, nb = n0 * n1 * n2, cr.num_bands
    i = np.arange(nq)
    neg = ((n2 - i // (n0 * n1)) % n2) * n0 * n1 + ((n1 - (i // n0) % n1) % n1) * n0 + (n0 - i % n0) % n0
    E = np.sort(rng.uniform(5e-4, 4e-3, (nq, nb)), axis=1)
    E[:, 1] = E[:, 0]
    E[i % 3 == 0, -1] = E[i % 3 == 0, -2]
    E = np.minimum(E, E[neg])
    E = np.sort(E, axis=1)
    U = np.linalg.qr(rng.normal(size=(nq, nb, nb)) + 1j * rng.normal(size=(nq, nb, nb)))[0]
    V = rng.normal(size=(nq, nb, 3)) * 5e-4
    half = i < neg
    U[neg[half]] = U[half].conj()
    V[neg[half]] = -V[half]
    own = i == neg
    U[own] = np.linalg.qr(rng.normal(size=(own.sum(), nb, nb)))[0]
    V[own] = 0.0
    return E, U, V, BandStructure.from_arrays(ctx, mesh, cr.reciprocal_cell, E, U, V)


@pytest.mark.parametrize("smearing", ["adaptive", "gaussian"])
@pytest.mark.parametrize("nat,mesh,nr3,window", [(1, (3, 2, 2), 1, False), (3, (3, 3, 2), 27, True), (5, (3, 2, 2), 8, False),
                                                 (5, (5, 4, 1), 125, True), (6, (3, 2, 2), 48, False), (8, (3, 2, 2), 57, True),
                                                 (9, (3, 2, 1), 27, False), (12, (3, 2, 1), 48, True),
                                                 (12, (3, 1, 1), 105, False), (13, (3, 1, 1), 9, False)])
def test_split_matches_fp64(ctx, nat, mesh, nr3, window, smearing):
    from phoebe_b200.core import Interaction3Ph, PhScatteringMatrix
    cr = _cell(nat)
    E, _, _, bands = _bands(ctx, cr, mesh, np.random.default_rng(nat))
    fc3 = _fc3(cr, nr3)
    T = np.array([C.kelvin_to_ry(t) for t in (100.0, 300.0, 600.0)])
    win = synth.q2_window(E, mesh) if window else None
    out = {}
    for precision in ("fp64", "split_fp16", "split_bf16"):
        v3 = Interaction3Ph(ctx, cr, fc3, precision=precision)
        sm = PhScatteringMatrix(v3, bands, T, smearing, 1e-4, window=win)
        out[precision] = sm.setup()
        if precision != "fp64":
            again = sm.setup(0, 1, finalize=False) + sm.setup(1, bands.nq, finalize=False)
            whole = sm.setup(finalize=False)
            # FP16 operands are scaled by the largest of a call: slices round differently
            np.testing.assert_allclose(again, whole, rtol=1e-5, atol=1e-8 * np.abs(whole).max())
        v3.close()
    A = out["fp64"]
    big = np.abs(A) > 1e-8 * np.abs(A).max()
    assert big.any()
    for precision in ("split_fp16", "split_bf16"):
        assert np.isfinite(out[precision]).all()
        assert (np.abs(out[precision] - A)[big] / np.abs(A)[big]).max() < 1e-5, precision
    bands.close()


def _fp64_against_oracle(ctx, nat, mesh, nr3, window, smearing):
    from phoebe_b200.core import Interaction3Ph, PhScatteringMatrix
    cr = _cell(nat)
    E, U, V, bands = _bands(ctx, cr, mesh, np.random.default_rng(nat))
    fc3 = _fc3(cr, nr3)
    T = np.array([C.kelvin_to_ry(t) for t in (100.0, 300.0)])
    win = synth.q2_window(E, mesh) if window else None
    v3 = Interaction3Ph(ctx, cr, fc3)
    A = PhScatteringMatrix(v3, bands, T, smearing, 1e-4, window=win).setup()
    v3.close()
    q = lattice.Mesh(cr, mesh).cartesian_coords()
    ref = oracle.Interaction3Ph(cr, fc3).linewidths(mesh, E, U, V, q, cr.reciprocal_cell, T, smearing, 1e-4, window=win)
    big = np.abs(ref) > 1e-8 * np.abs(ref).max()
    assert big.any()
    assert (np.abs(A - ref)[big] / np.abs(ref)[big]).max() < 1e-10
    bands.close()


@pytest.mark.parametrize("smearing", ["adaptive", "gaussian"])
@pytest.mark.parametrize("nat,mesh,nr3,window", [(1, (3, 2, 2), 1, False), (2, (5, 4, 1), 4, True), (3, (3, 3, 2), 27, False),
                                                 (5, (3, 2, 2), 67, True), (5, (3, 2, 1), 130, False),
                                                 (5, (3, 1, 1), 343, True)])
def test_fp64_matches_oracle(ctx, nat, mesh, nr3, window, smearing):
    _fp64_against_oracle(ctx, nat, mesh, nr3, window, smearing)


@pytest.mark.parametrize("smearing", ["adaptive", "gaussian"])
@pytest.mark.parametrize("nat,mesh,nr3,window", [(1, (3, 2, 2), 1, False), (1, (5, 4, 1), 343, True), (2, (5, 4, 1), 4, True),
                                                 (2, (5, 4, 1), 49, True), (2, (5, 4, 1), 50, True), (2, (3, 2, 2), 250, True),
                                                 (3, (3, 3, 2), 27, False), (4, (5, 4, 1), 1, True), (5, (3, 2, 2), 67, True),
                                                 (5, (3, 2, 1), 130, False)])
def test_fp64_many_branch_matches_oracle(ctx, monkeypatch, nat, mesh, nr3, window, smearing):
    """The same on the many-branch builder, which problems as small as these reach only when forced: the
    tensor-pipe kernel, and wide.cu's up to 6 branches (6 branches: fewer than 50 R3)."""
    monkeypatch.setenv("PHX_WIDE", "1")
    _fp64_against_oracle(ctx, nat, mesh, nr3, window, smearing)


# items of 16 q1 and a q2, blocks of 4 q1 and a q2, on 148 SMs
@pytest.mark.parametrize("nat,mesh,q2,many_branch", [
    (1, (8, 8, 2), 36, False), (1, (8, 8, 2), 37, True), (2, (8, 8, 2), 36, False), (2, (8, 8, 2), 37, True),
    (3, (5, 5, 3), 29, False), (3, (5, 5, 3), 30, True), (4, (4, 4, 2), 18, False), (4, (4, 4, 2), 19, True),
    (5, (3, 3, 1), 9, False), (5, (4, 4, 2), 18, False), (5, (4, 4, 2), 19, True)])
def test_fp64_route_by_size(ctx, monkeypatch, nat, mesh, q2, many_branch):
    """Little work stays on the shared-memory builder (no pair events); both sides of the line agree with
    the forced many-branch builder."""
    from phoebe_b200.core import Interaction3Ph, PhScatteringMatrix
    cr = _cell(nat)
    E, _, _, bands = _bands(ctx, cr, mesh, np.random.default_rng(nat))
    v3 = Interaction3Ph(ctx, cr, _fc3(cr, 9))
    sm = PhScatteringMatrix(v3, bands, [C.kelvin_to_ry(300.0)], "adaptive", 0.0,
                            window=synth.q2_window(E, mesh) if nat == 2 else None)
    A = sm.setup(0, q2, finalize=False)
    assert (sm.stats.pair_launches > 0) == many_branch
    monkeypatch.setenv("PHX_WIDE", "1")
    B = sm.setup(0, q2, finalize=False)
    assert np.abs(B).max() > 0
    np.testing.assert_allclose(A, B, rtol=1e-10, atol=1e-14 * np.abs(B).max())
    v3.close()
    bands.close()


@pytest.mark.parametrize("precision", ["fp64", "split_fp16"])
@pytest.mark.parametrize("nat,mesh,window", [(1, (3, 2, 2), False), (3, (4, 4, 2), True), (3, (5, 7, 1), False),
                                             (5, (3, 3, 2), True)])
def test_isotopes_in_slots_match_oracle(ctx, monkeypatch, nat, mesh, window, precision):
    """Isotope rates of the many-branch builder, a slot per q2 on these meshes: one tile of 32 q1,
    exactly one, and a remainder; slices of q2 add up.  FP64 at 1e-10, split at its 1e-5."""
    from phoebe_b200.core import Interaction3Ph, PhScatteringMatrix, isotope_coupling
    monkeypatch.setenv("PHX_WIDE", "1")
    cr = _cell(nat)
    E, U, V, bands = _bands(ctx, cr, mesh, np.random.default_rng(nat))
    fc3 = _fc3(cr, 5)
    fc3.D3 *= 1e-3   # rates of the size of the isotopes'
    T = np.array([C.kelvin_to_ry(t) for t in (100.0, 300.0)])
    win = synth.q2_window(E, mesh) if window else None
    g = isotope_coupling(cr, np.linspace(1e-2, 3e-2, nat))
    v3 = Interaction3Ph(ctx, cr, fc3, precision=precision)
    sm = PhScatteringMatrix(v3, bands, T, "adaptive", 0.0, window=win, isotope_coupling=g)
    A = sm.setup(finalize=False)
    parts = sm.setup(0, 2, finalize=False) + sm.setup(2, bands.nq, finalize=False)
    np.testing.assert_allclose(parts, A, rtol=1e-12 if precision == "fp64" else 1e-5, atol=1e-8 * np.abs(A).max())
    v3.close()
    q = lattice.Mesh(cr, mesh).cartesian_coords()
    ref, without = (oracle.Interaction3Ph(cr, fc3).linewidths(mesh, E, U, V, q, cr.reciprocal_cell, T, "adaptive", 0.0,
                                                              window=win, finalize=False, isotope_coupling=i)
                    for i in (g, None))
    assert (ref > 1.01 * without).any()
    tol = 1e-10 if precision == "fp64" else 1e-5
    big = np.abs(ref) > 1e-8 * np.abs(ref).max()
    assert (np.abs(A - ref)[big] / np.abs(ref)[big]).max() < tol
    bands.close()
