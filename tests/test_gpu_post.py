"""Post-processing kernels at the sizes where their work splits change.

Refinement: one block of 16 warps per pose, 4 atoms per warp at a time (so
groups of 4 and rounds of 64 atoms), receptor neighbours in tiles of 32, the
intra pairs spread over the block and summed per run of one second atom.
Sizes: no intra pairs, group and round remainders, the largest ligand, the
most intra pairs; receptors with no atom in reach, fewer than a tile and
several tiles of neighbours.
"""
import numpy as np
import pytest

import oracle_lib as O
from conftest import has_gpu

pytestmark = pytest.mark.gpu


def _env(rec_atoms, radius, na, nt, seed=5):
    if not has_gpu():
        pytest.skip("needs a CUDA device")
    import vdock
    from vdock import synth
    xyz, xs = synth.receptor(rec_atoms, radius, 9) if rec_atoms else (np.zeros((0, 3)), np.zeros(0, np.int32))
    lig = synth.ligand(na, nt, seed)
    ctx, orc = vdock.Context(), O.Oracle()
    for o in (ctx, orc):
        o.set_receptor(xyz, xs)
        o.set_box([0.0, 0.0, 0.0], [34.0] * 3)
        o.build_grids(list(range(17)))
    return ctx, orc, lig, ctx.add_ligand(lig), orc.add_ligand(lig), synth


# (receptor atoms, their ball's radius, ligand atoms, torsions): the densest
# ball holds ~0.02 atoms per A^3, about 90 neighbours per cell
REFINE = [(2000, 40.0, 2, 0), (2000, 40.0, 5, 1), (0, 1.0, 17, 4), (1200, 24.0, 32, 6), (1200, 24.0, 33, 9),
          (2000, 40.0, 64, 12), (2000, 40.0, 65, 15), (2000, 40.0, 128, 3), (2000, 40.0, 100, 20)]


@pytest.mark.parametrize("rec_atoms,radius,na,nt", REFINE)
def test_refinement_sizes(rec_atoms, radius, na, nt):
    """Each returned energy is its pose's direct-sum energy (the tolerance of
    test_refine_matches_oracle_distribution), none is above its start's, and
    one optimiser step from the same starts gives the oracle's energies: a
    step is start + alpha * (-gradient) with alpha a power of two, so FP32
    rounding enters once and the same tolerance holds wherever the line
    search stops at the same alpha; a tenth of the poses may not (an Armijo
    test within rounding of its bound)."""
    ctx, orc, lig, lc, lo, synth = _env(rec_atoms, radius, na, nt)
    starts = synth.random_poses(21, ctx.ntors[lc], -2.0, 2.0, seed=na)
    _, starts, _ = ctx.local_opt(lc, starts, 20)
    _, b, en = orc.grid_info()

    def direct(p):
        return orc.eval_deriv(lo, p.astype(np.float64), v=(1000, 1000, 1000), slope=1e6, noncache=True)[0]

    e, p = ctx.refine(lc, starts, 15)
    n_in = 0
    for i in range(len(starts)):
        x = orc.coords(lo, p[i].astype(np.float64), lig["n_atoms"])
        if not (e[i] < 1e30 and np.all(x > b) and np.all(x < en)):
            continue
        n_in += 1
        ref = direct(p[i])
        assert abs(ref - e[i]) <= 2e-3 * max(1.0, abs(ref)), (i, ref, e[i])
        xs = orc.coords(lo, starts[i].astype(np.float64), lig["n_atoms"])
        if np.all(xs > b) and np.all(xs < en):
            s = direct(starts[i])
            assert e[i] <= s + 2e-3 * max(1.0, abs(s)), (i, s, e[i])
    assert n_in >= 10
    e1, _ = ctx.refine(lc, starts, 1)
    same = checked = 0
    for i in range(len(starts)):
        r, _, _ = orc.refine(lo, starts[i].astype(np.float64), 1)
        if r < 1e30 and e1[i] < 1e30:
            checked += 1
            same += abs(r - e1[i]) <= 2e-3 * max(1.0, abs(r))
    assert checked >= 10 and same >= 0.9 * checked, (same, checked)


def test_non_finite_poses_stay_in_bounds():
    """Positions and torsions that are infinite or not a number have no
    receptor cell: they take an edge cell, and the poses beside them are
    refined and scored to the same bits as without them."""
    ctx, _, lig, lc, _, synth = _env(1200, 24.0, 33, 9)
    starts = synth.random_poses(12, ctx.ntors[lc], -2.0, 2.0, seed=4)
    e0, p0 = ctx.refine(lc, starts, 5)
    s0 = ctx.score(lc, starts)
    bad = starts.copy()
    rows = {2: (0, np.nan), 5: (1, np.inf), 7: (2, -np.inf), 8: (7, np.nan), 10: (0, 3e38)}
    for i, (k, v) in rows.items():
        bad[i, k] = v
    e1, p1 = ctx.refine(lc, bad, 5)
    s1 = ctx.score(lc, bad)
    keep = [i for i in range(len(starts)) if i not in rows]
    assert np.array_equal(e0[keep], e1[keep]) and np.array_equal(p0[keep], p1[keep])
    for a, b in zip(s0, s1):
        assert np.array_equal(np.asarray(a)[keep], np.asarray(b)[keep])
