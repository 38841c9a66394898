"""Pose batches where the choice of kernel and tile changes for ligands of many pairs: few bodies (a warp per pose between
tiles), tiles of 16 poses on 16 warps, a largest tile that an SM holds once.  Energies and gradients against the oracle,
with the tolerances of test_gpu_tiles; coordinates the same bits however many poses a call has."""
import numpy as np
import pytest

import oracle_lib as O
from conftest import has_gpu

pytestmark = pytest.mark.gpu


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
        o.set_box([0.0, 0.0, 0.0], [44.0] * 3)
        o.build_grids(list(range(17)))
    return ctx, orc, synth, torch.cuda.get_device_properties(0).multi_processor_count


# poses per SM on either side of each line of the rule (and one more or less)
@pytest.mark.parametrize("na,nt,per_sm", [(50, 5, (10, 15.9, 16, 28)), (60, 3, (12, 23.9, 24, 31.9)), (80, 2, (10, 16, 27.9, 28)),
                                          (128, 3, (15.9, 17.9, 18, 24, 50, 63.9, 64)), (80, 6, (7.9, 8.1, 24)),
                                          (90, 32, (31.9, 50, 64)), (100, 12, (47, 64))])
def test_rule_edges(env, na, nt, per_sm):
    ctx, orc, synth, sms = env
    lig = synth.ligand(na, nt, 3)
    lc, lo = ctx.add_ligand(lig), orc.add_ligand(lig)
    npts, b, en = orc.grid_info()
    cell = (en - b) / (npts - 1)
    poses = synth.random_poses(int(max(per_sm) * sms) + 2, nt, -2.0, 2.0, seed=na)
    xyz = ctx.pose_coords(lc, poses)
    rng = np.random.default_rng(na)
    checked = 0
    for per in per_sm:
        for n in (int(per * sms) - 1, int(per * sms) + 1):
            assert np.array_equal(ctx.pose_coords(lc, poses[:n]), xyz[:n]), n
            e, g = ctx.energy_grad(lc, poses[:n])
            e0 = ctx.energy(lc, poses[:n])
            for i in sorted(set(rng.integers(0, n, size=3)) | {0, n - 1}):
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
    assert checked >= 3
