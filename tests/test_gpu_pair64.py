"""The FP64 pair kernel of the 6-branch cells (tensor-pipe R3 transform) against
the oracle on identical band structures, at the edges of its tiles: meshes
smaller than a warp's 8 q1 and than a block's tile, q1 counts that are no
multiple of either, R3 counts around the K step of 4 and beyond one ring stage,
and the largest R3 count the path takes (fewer warps per block); larger ones are
refused.  The stored matrix is the same in every build, and the slots of coarse
meshes and of short slices are those that pay.  1e-10 is the
bar of the other FP64 linewidth tests (sums of ~1e5 terms, each with a few
rounding errors of 1e-16, and the cancellation of the R3 sum)."""
import numpy as np
import pytest

import oracle
from phoebe_b200 import constants as C
from phoebe_b200 import lattice, synth

pytestmark = pytest.mark.gpu


def _fc3(cr, nr3):
    """A random real tensor on one R2 and nr3 R3 vectors (no sum rule: the kernels need none)."""
    R, _ = synth.lattice_cube(cr, 3 if nr3 <= 343 else 6)
    rng = np.random.default_rng(nr3)
    o = np.argsort(np.linalg.norm(R, axis=1), kind="stable")
    D3 = rng.normal(size=(6, 6, 6, nr3, 1)) * 0.05
    nat = cr.num_atoms
    return synth.FC3(D3, R[o[1:2]], R[o[:nr3]], np.ones((1, nat, nat)), np.ones((nr3, nat, nat)), nr3)


def _bands(ctx, cr, mesh):
    from phoebe_b200.core import PhononH0
    h0 = PhononH0(ctx, cr, synth.diamond_fc2(cr))
    bands = h0.populate(mesh, withVelocities=True)
    h0.close()
    return bands


def _close(a, b, rtol):
    scale = np.abs(b).max()
    assert scale > 0
    big = np.abs(b) > 1e-6 * scale
    assert (np.abs(a - b)[big] / np.abs(b)[big]).max() < rtol
    assert np.abs(a - b)[~big].max(initial=0.0) < rtol * 1e-6 * scale


@pytest.mark.parametrize("smearing,temps", [("adaptive", (100.0, 300.0, 600.0, 900.0)), ("gaussian", (300.0,))])
@pytest.mark.parametrize("mesh,nr3", [((2, 2, 1), 1), ((3, 3, 1), 4), ((4, 4, 4), 5), ((5, 3, 5), 48),
                                      ((3, 3, 3), 49), ((5, 4, 3), 97), ((2, 3, 2), 262)])
def test_linewidths_at_tile_edges(ctx, mesh, nr3, smearing, temps):
    from phoebe_b200.core import Interaction3Ph, PhScatteringMatrix
    cr = synth.diamond_crystal()
    fc3 = _fc3(cr, nr3)
    bands = _bands(ctx, cr, mesh)
    E, U, vg = bands.get()
    T = np.array([C.kelvin_to_ry(t) for t in temps])
    v3 = Interaction3Ph(ctx, cr, fc3)
    sm = PhScatteringMatrix(v3, bands, T, smearing, 0.3 / C.ryToTHz)
    A = sm.setup()
    m = lattice.Mesh(cr, mesh)
    ref = oracle.Interaction3Ph(cr, fc3).linewidths(mesh, E, U, vg, m.cartesian_coords(), cr.reciprocal_cell, T,
                                                    smearing, 0.3 / C.ryToTHz)
    _close(A, ref, 1e-10)
    # a rank's q2 slice of one point
    part = sm.setup(1, 2, finalize=False)
    rest = [sm.setup(0, 1, finalize=False), sm.setup(2, bands.nq, finalize=False)]
    whole = sm.setup(finalize=False)
    np.testing.assert_allclose(part + rest[0] + rest[1], whole, rtol=1e-12, atol=1e-14 * np.abs(whole).max())
    v3.close()
    bands.close()


@pytest.mark.parametrize("nr3", [263, 1380, 1381, 1400])
def test_too_many_r3_vectors_are_refused(ctx, nr3):
    """Past 262 R3 vectors the path returns an error, also past 1380, where no warp's phases fit."""
    from phoebe_b200.core import Interaction3Ph, PhScatteringMatrix
    cr = synth.diamond_crystal()
    bands = _bands(ctx, cr, (2, 2, 1))
    v3 = Interaction3Ph(ctx, cr, _fc3(cr, nr3))
    T = [C.kelvin_to_ry(300.0)]
    sm = PhScatteringMatrix(v3, bands, T)
    with pytest.raises(RuntimeError, match="too many R3 vectors"):
        sm.setup()
    with pytest.raises(RuntimeError, match="too many R3 vectors"):
        sm.dot(np.zeros((1, 3, sm.num_states)))
    with pytest.raises(RuntimeError, match="too many R3 vectors"):
        PhScatteringMatrix(v3, bands, T, in_memory=True).setup()
    v3.close()
    bands.close()


@pytest.mark.parametrize("smearing", ["adaptive", "gaussian"])
def test_matrix_modes_with_degenerate_points(ctx, diamond, smearing):
    """Stored matrix and matrix-free product; the diamond's symmetry points have degenerate
    blocks of b1, b2 and b3, some across the kernel's pairs of b2."""
    from phoebe_b200.core import Interaction3Ph, PhScatteringMatrix
    cr, mesh = diamond["crystal"], (3, 4, 3)
    bands = _bands(ctx, cr, mesh)
    E, U, vg = bands.get()
    T = C.kelvin_to_ry(300.0)
    sigma = 0.5 / C.ryToTHz
    ref = oracle.Interaction3Ph(cr, diamond["fc3"])
    q = lattice.Mesh(cr, mesh).cartesian_coords()
    mat, lw = ref.scattering_matrix(mesh, E, U, vg, q, cr.reciprocal_cell, T, smearing, sigma)
    v3 = Interaction3Ph(ctx, cr, diamond["fc3"])
    sm = PhScatteringMatrix(v3, bands, [T], smearing, sigma, in_memory=True)
    _close(sm.setup(), lw[None], 1e-10)
    _close(sm.getMatrixRows(0, sm.num_states), mat, 1e-10)
    x = np.random.default_rng(1).normal(size=(2, 1, 3, sm.num_states))
    free = PhScatteringMatrix(v3, bands, [T], smearing, sigma)
    y = free.dot(x)
    np.testing.assert_allclose(y, sm.dot(x), rtol=0, atol=1e-11 * np.abs(y).max())
    sm.close()
    v3.close()
    bands.close()


@pytest.mark.parametrize("mesh", [(4, 4, 4), (9, 9, 9), (11, 10, 12)])
def test_stored_matrix_is_the_same_every_time(ctx, diamond, mesh):
    """One "+" and one "-" addition onto zero for each element, whatever the order of the blocks (one
    wave of them and several), also where the bands of q2 are degenerate."""
    from phoebe_b200.core import Interaction3Ph, PhScatteringMatrix
    bands = _bands(ctx, diamond["crystal"], mesh)
    v3 = Interaction3Ph(ctx, diamond["crystal"], diamond["fc3"])
    sm = PhScatteringMatrix(v3, bands, [C.kelvin_to_ry(300.0)], "gaussian", 0.5 / C.ryToTHz, in_memory=True)
    diag, rows = sm.setup(), sm.getMatrixRows(0, sm.num_states)
    for _ in range(8):
        np.testing.assert_array_equal(sm.setup(), diag)
        np.testing.assert_array_equal(sm.getMatrixRows(0, sm.num_states), rows)
    sm.close()
    v3.close()
    bands.close()


# slots of 148 SMs: a q2 each where that is one wave or less, two (split) and three (FP64) q2 at
# 7x5x4, whose tiles are 2 of 128 and 3 of 64 q1
@pytest.mark.parametrize("mesh,slots64,slots16", [((2, 1, 1), 2, 2), ((3, 3, 3), 27, 27), ((7, 5, 4), 47, 70)])
def test_coarse_meshes_fill_the_chip(ctx, diamond, mesh, slots64, slots16):
    """A q2 range too short to be tuned takes as many slots as fill the SMs; the split path's
    linewidths keep its 1e-5 bar against FP64, whose own slots sum in another order (1e-12)."""
    from phoebe_b200.core import Interaction3Ph, PhScatteringMatrix
    cr = diamond["crystal"]
    bands = _bands(ctx, cr, mesh)
    T = np.array([C.kelvin_to_ry(t) for t in (100.0, 300.0)])
    out = {}
    for precision, slots in (("fp64", slots64), ("split_fp16", slots16)):
        v3 = Interaction3Ph(ctx, cr, diamond["fc3"], precision=precision)
        sm = PhScatteringMatrix(v3, bands, T, "adaptive")
        out[precision] = sm.setup()
        assert sm.stats.plan_slots == slots
        half = sm.setup(0, bands.nq // 2, finalize=False) + sm.setup(bands.nq // 2, bands.nq, finalize=False)
        whole = sm.setup(finalize=False)
        np.testing.assert_allclose(half, whole, rtol=1e-12 if precision == "fp64" else 1e-6,
                                   atol=1e-12 * np.abs(whole).max())
        v3.close()
    if bands.nq > 2:
        _close(out["split_fp16"], out["fp64"], 1e-5)
    bands.close()


@pytest.mark.parametrize("mesh,q2,slots", [((17, 17, 17), 32, 7), ((20, 20, 20), 24, 7), ((20, 20, 20), 32, 7),
                                           ((24, 24, 24), 8, 7)])
def test_short_slices_keep_blocks_for_several_waves(ctx, diamond, mesh, q2, slots):
    """A slice of a few q2 of a fine mesh: one wave of long blocks waits for its slowest tile
    (39 to 108 tiles of the split kernel), so the slots stay at the untuned plan's 7."""
    from phoebe_b200.core import Interaction3Ph, PhScatteringMatrix
    bands = _bands(ctx, diamond["crystal"], mesh)
    v3 = Interaction3Ph(ctx, diamond["crystal"], diamond["fc3"], precision="split_fp16")
    sm = PhScatteringMatrix(v3, bands, [C.kelvin_to_ry(300.0)])
    sm.setup(0, q2, finalize=False)
    assert sm.stats.plan_slots == slots
    v3.close()
    bands.close()
