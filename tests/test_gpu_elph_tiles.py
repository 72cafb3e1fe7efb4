"""Tiles of the electron-phonon pair kernel: final states in eights per initial
state, Rp and Re in fours, columns in eights and 32s, and the sizes where one
final state is taken at a time, from a list or without one, against the oracle."""
import numpy as np
import pytest

import oracle
from phoebe_b200 import constants as C
from phoebe_b200 import lattice, synth

pytestmark = pytest.mark.gpu


def _crystal(nat):
    p = synth.perovskite_crystal()
    masses = (137.0, 48.0, 16.0, 16.0)[:nat]
    return lattice.Crystal(p.direct_cell, p.positions[:nat], np.arange(nat), np.array(masses) * C.massAmuToRy)


def _compare(ctx, nat, nw, ce, cp, kmesh, qmesh, window, smearing, nk1, precision):
    """The linewidths of nk1 initial states against the oracle; returns the call's stats."""
    from phoebe_b200.core import ElectronH0Wannier, ElScatteringMatrix, InteractionElPhWan, PhononH0
    cr = _crystal(nat)
    Rh, degh, H = synth.wannier_hamiltonian(cr, nw, 1)
    Re, degE, Rp, degP, g = synth.elph_coupling(cr, ce, cp, 3 * nat, nw)
    a = cr.direct_cell[0, 0]
    k = 5.0 * C.distanceBohrToAng ** 2 / C.energyRyToEv
    shells = [(r * a, k, None) for r in (0.5, 0.5 ** 0.5, 0.75 ** 0.5, 1.0, 2.0 ** 0.5)]
    wan = ElectronH0Wannier(ctx, cr, Rh, degh, H)
    el = wan.populate(kmesh, withVelocities=True)
    h0 = PhononH0(ctx, cr, synth.spring_fc2(cr, shells))
    ph = h0.populate(qmesh, withVelocities=False)
    Ek, Uk, vk = el.get()
    Eq, evq, _ = ph.get(velocities=False)
    mu = float(np.median(Ek))
    win = 1.0 + 2.0 * np.abs(Ek).max() if window == "all" else 0.6 * float(Ek.std())
    lo, hi = synth.active_window(Ek, mu, win)
    k1 = np.linspace(0, np.prod(kmesh) - 1, nk1).astype(np.int32)
    temps = np.array([C.kelvin_to_ry(300.0), C.kelvin_to_ry(900.0)])
    sigma = 0.05
    gpu = InteractionElPhWan(ctx, Re, degE, Rp, degP, g)
    gpu.setPrecision(precision)
    sm = ElScatteringMatrix(gpu, el, ph, temps, mu, win, smearing, sigma)
    A = sm.setup(k1)
    ref = oracle.InteractionElPhWan(Re, degE, Rp, degP, g)
    kc = lattice.Mesh(cr, kmesh).cartesian_coords()
    B = oracle.el_linewidths(ref, kmesh, qmesh, Ek, Uk, vk, lo, hi, Eq, evq, kc, cr.reciprocal_cell, k1, temps, mu,
                             smearing, sigma, 1.0 / np.prod(qmesh))
    assert np.abs(B).max() > 0
    # FP64: sums of at most 343 x 25 terms, 1e-10 as for the couplings; split: three BF16
    # products of 16-bit pieces, 2^-16 of the largest terms, 1e-5 of the strongest state
    tol = 1e-10 if precision == "fp64" else 1e-5
    big = np.abs(B) > (1e-9 if precision == "fp64" else 1e-2) * np.abs(B).max()
    assert (np.abs(A - B)[big] / np.abs(B)[big]).max() < tol
    assert np.abs(A - B).max() < tol * np.abs(B).max()
    for h in (gpu, ph, h0, el, wan):
        h.close()
    return sm.stats


# nat (3 nat branches), nw, ncell of Re and Rp, k mesh, q mesh, bands in the window, smearing, k1.
# 4 atoms with all 8 bands active are past the tile's shared memory; with 5 they are within.
# 21 and 17 k1 leave a second batch of at most 8.
@pytest.mark.parametrize("nat,nw,ce,cp,kmesh,qmesh,window,smearing,nk1", [
    (1, 1, 1, 1, (3, 3, 3), (3, 3, 3), "all", "gaussian", 3),
    (1, 5, 1, 2, (4, 2, 6), (2, 2, 3), "some", "adaptive", 21),
    (2, 3, 2, 1, (5, 5, 3), (5, 5, 3), "all", "adaptive", 17),
    (2, 8, 1, 0, (6, 4, 2), (3, 2, 2), "some", "gaussian", 16),
    (4, 8, 1, 1, (4, 4, 2), (2, 2, 2), "some", "adaptive", 9),
    (4, 8, 1, 1, (4, 4, 2), (2, 2, 2), "all", "adaptive", 9),
    (4, 8, 0, 1, (4, 4, 2), (2, 2, 2), "all", "gaussian", 2),
])
@pytest.mark.parametrize("precision", ["fp64", "split_bf16"])
def test_el_linewidths_tiles(ctx, nat, nw, ce, cp, kmesh, qmesh, window, smearing, nk1, precision):
    _compare(ctx, nat, nw, ce, cp, kmesh, qmesh, window, smearing, nk1, precision)


# Split: up to 4096 final states of a batch a block for each, none listed; past that tiles of 8, or past 8192
# blocks of one state where the buffers of a tile leave few of them on an SM (6 branches, 8 bands) or do not
# fit (12).  FP64: tiles, but blocks of one state with a tile per SM and few Rp, or where tiles do not fit.
# The launches tell: one more per batch with a list.
@pytest.mark.parametrize("nat,nw,ce,cp,kmesh,qmesh,window,smearing,nk1,precision,launches", [
    (1, 5, 1, 1, (8, 8, 8), (8, 8, 8), "some", "adaptive", 8, "split_bf16", 11),
    (1, 5, 1, 1, (8, 8, 8), (8, 8, 8), "some", "adaptive", 9, "split_bf16", 12),
    (2, 8, 0, 1, (9, 8, 8), (9, 8, 8), "all", "gaussian", 14, "split_bf16", 11),
    (2, 8, 1, 1, (9, 8, 8), (9, 8, 8), "all", "gaussian", 17, "split_bf16", 19),
    (4, 8, 0, 0, (9, 8, 8), (9, 8, 8), "all", "adaptive", 15, "split_bf16", 12),
    (2, 8, 0, 1, (9, 8, 8), (9, 8, 8), "all", "adaptive", 8, "fp64", 8),
    (4, 8, 0, 1, (4, 4, 2), (2, 2, 2), "all", "gaussian", 3, "fp64", 7),
])
def test_el_linewidths_routes(ctx, nat, nw, ce, cp, kmesh, qmesh, window, smearing, nk1, precision, launches):
    stats = _compare(ctx, nat, nw, ce, cp, kmesh, qmesh, window, smearing, nk1, precision)
    assert stats.kernel_launches == launches
