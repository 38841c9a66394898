"""Post-processing whose split follows the amount of work (refinement on 16, 8, 4 or 1 warps a pose, clustering and scoring
on as many warps as a ligand has chains): a pose's result has the same bits whatever stands beside it."""
import numpy as np
import pytest

from conftest import has_gpu

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def env():
    if not has_gpu():
        pytest.skip("needs a CUDA device")
    import torch
    import vdock
    from vdock import synth
    ctx = vdock.Context()
    ctx.set_receptor(*synth.receptor(1500, 35.0, 9))
    ctx.set_box([0.0, 0.0, 0.0], [28.0] * 3)
    ctx.build_grids(list(range(17)))
    return vdock, ctx, synth, torch.cuda.get_device_properties(0).multi_processor_count


@pytest.mark.parametrize("na,nt", [(2, 0), (16, 3), (17, 3), (28, 6), (29, 6), (66, 15)])
def test_refinement(env, na, nt):
    _, ctx, synth, sms = env
    lig = ctx.add_ligand(synth.ligand(na, nt, 5))
    poses = synth.random_poses(61 * sms, nt, -4.0, 4.0, seed=na)
    poses[3, 0] = np.nan
    ref_e, ref_p = ctx.refine(lig, poses[:64], 3)  # 16 warps a pose
    for n in (3 * sms, 7 * sms, 11 * sms, 31 * sms, 41 * sms, 61 * sms):
        e, p = ctx.refine(lig, poses[:n], 3)
        assert np.array_equal(e[:64], ref_e, equal_nan=True) and np.array_equal(p[:64], ref_p, equal_nan=True), n


@pytest.mark.parametrize("chains,ligands", [(1, 700), (2, 300), (5, 300), (16, 120), (21, 40), (100, 12)])
def test_docking_batches(env, chains, ligands):
    vd, ctx, synth, _ = env
    ids = [ctx.add_ligand(synth.ligand(6 + i % 25, i % 4, i)) for i in range(ligands)]
    sp = vd.search_params(seed=3, n_chains=chains, search_depth=1, max_bfgs_steps=4, refine=1, num_modes=20, energy_range=1e6)
    batch = ctx.dock_batched(ids, sp)
    for i in range(0, ligands, max(1, ligands // 12)):
        one = ctx.dock_plain(ids[i], sp)
        for k in ("energy", "pose", "rmsd_lb", "rmsd_ub"):
            assert np.array_equal(one[k], batch[i][k]), (i, k)
        assert one["bfgs_evals"] == batch[i]["bfgs_evals"] and len(one["energy"]) <= chains
