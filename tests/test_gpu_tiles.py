"""Pose batches evaluated in tiles (1, 4, 8, 16 or 32 poses per block) at the
numbers of poses where the tile changes, with a short last tile, for ligands
with no pairs, few, odd numbers and the most, bodies past a tile's slots and
atoms at the limit.

Energies and gradients against the oracle (1e-3 kcal/mol inside the box and
1e-3 of |g|_inf, the tolerances of test_gpu_limits), gradients where no atom
is within 1e-5 A of a cell face or outside the box; coordinates bit for bit
the same however many poses a call has, in tiles and in the warp-per-pose
kernel that small ligands take below 64 poses per SM.
"""
import numpy as np
import pytest

import oracle_lib as O
from conftest import has_gpu

pytestmark = pytest.mark.gpu

SIZES = [(2, 0), (12, 2), (33, 9), (37, 9), (41, 10), (90, 32), (100, 20), (128, 3), (70, 48)]


@pytest.fixture(scope="module")
def env():
    if not has_gpu():
        pytest.skip("needs a CUDA device")
    import torch
    import vdock
    from vdock import synth
    ctx, orc = vdock.Context(), O.Oracle()
    for o in (ctx, orc):
        o.set_receptor(*synth.receptor(1000, 30.0, 3))
        o.set_box([0.0, 0.0, 0.0], [36.0] * 3)
        o.build_grids(list(range(17)))
    return ctx, orc, synth, torch.cuda.get_device_properties(0).multi_processor_count


@pytest.mark.parametrize("na,nt", SIZES)
def test_tiles_match_the_oracle(env, na, nt):
    ctx, orc, synth, sms = env
    lig = synth.ligand(na, nt, 5)
    lc, lo = ctx.add_ligand(lig), orc.add_ligand(lig)
    npts, b, en = orc.grid_info()
    cell = (en - b) / (npts - 1)
    poses = synth.random_poses(64 * sms + 3, ctx.ntors[lc], -3.0, 3.0, seed=na)
    xyz = ctx.pose_coords(lc, poses)
    rng = np.random.default_rng(na)
    checked = 0
    for n in (1, 3, 3 * sms + 1, 16 * sms + 5, 32 * sms + 7, len(poses)):
        assert np.array_equal(ctx.pose_coords(lc, poses[:n]), xyz[:n]), n
        e, g = ctx.energy_grad(lc, poses[:n])
        e0 = ctx.energy(lc, poses[:n])
        for i in sorted(set(rng.integers(0, n, size=5)) | {0, n - 1}):
            p = poses[i].astype(np.float64)
            e_ref, g_ref = orc.eval_deriv(lo, p)
            x = orc.coords(lo, p, lig["n_atoms"])
            s = (x - b) / cell
            inside = np.all((x > b + 1e-4) & (x < en - 1e-4))
            tol = 1e-3 if inside else 1e-4 * abs(e_ref) + 1e-3
            assert abs(e[i] - e_ref) <= tol and abs(e0[i] - e_ref) <= tol, (n, i, e[i], e0[i], e_ref)
            if inside and np.abs(s - np.round(s)).min() > 1e-5 / cell.min():
                checked += 1
                assert np.abs(g[i] - g_ref).max() <= 1e-3 * max(1.0, np.abs(g_ref).max()), (n, i)
    assert checked >= 10
