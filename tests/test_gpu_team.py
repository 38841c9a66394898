"""Docking chains evaluated by a team of warps (few chains, shape 5) against
one warp per chain (shape 1): bit-identical chains, modes and evaluation
counts.  Pair energies are added in the single warp's order and pair forces
are integer sums, so nothing may differ.  Ligands: no intra pairs, fewer
schedule entries than helper warps, more than one round of them, atoms past
one and two per lane, the largest accepted; both searches; the plain form,
the batched form over ligands of different sizes, and a call with no
Monte-Carlo step.  Local optimisation picks its kernel by the number of poses:
a pose's result may not depend on how many others there are.
"""
import numpy as np
import pytest

from conftest import has_gpu

pytestmark = pytest.mark.gpu

SIZES = [(2, 0), (10, 0), (14, 3), (32, 6), (33, 9), (65, 12), (100, 20), (128, 3)]


@pytest.fixture(scope="module")
def env():
    if not has_gpu():
        pytest.skip("needs a CUDA device")
    import vdock
    from vdock import synth
    ctx = vdock.Context()
    ctx.set_receptor(*synth.receptor(1500, 35.0, 3))
    ctx.set_box([0.0, 0.0, 0.0], [20.0] * 3)
    ctx.build_grids(synth.TYPES8)
    return vdock, ctx, [ctx.add_ligand(synth.ligand(na, nt, 5)) for na, nt in SIZES]


@pytest.mark.parametrize("dense", [0, 1])
@pytest.mark.parametrize("i", range(len(SIZES)))
def test_team_chains_equal_single_warp_chains(env, i, dense):
    vd, ctx, ids = env
    out = []
    for shape in (5, 1, 0):
        sp = vd.search_params(seed=7, n_chains=37, search_depth=2, max_bfgs_steps=8, launch_shape=shape, dense_bfgs=dense)
        out.append(ctx.mc_chains(ids[i], sp))
        assert ctx.stats()["dock_warps_per_block"] == (4 if shape == 1 else 1)
    for p, e, ev in out[1:]:
        assert np.array_equal(p, out[0][0]) and np.array_equal(e, out[0][1]) and ev == out[0][2]


@pytest.mark.parametrize("dense,depth,visited", [(0, 3, 0), (1, 2, 0), (0, 2, 1), (0, -1, 0)])
def test_team_batches_equal_single_warp_batches(env, dense, depth, visited):
    vd, ctx, ids = env
    out = []
    for shape in (5, 1):
        sp = vd.search_params(seed=9, n_chains=24, search_depth=depth, max_bfgs_steps=6, launch_shape=shape,
                              dense_bfgs=dense, visited_history=visited)
        out.append(ctx.dock_batched(ids, sp))
        assert ctx.stats()["dock_warps_per_block"] == (4 if shape == 1 else 1)
    for a, b in zip(*out):
        assert a["bfgs_evals"] == b["bfgs_evals"]
        assert np.array_equal(a["energy"], b["energy"]) and np.array_equal(a["pose"], b["pose"])


@pytest.mark.parametrize("i", [0, 2, 4, 6])
def test_local_optimisation_does_not_depend_on_the_number_of_poses(env, i):
    import torch
    from vdock import synth
    vd, ctx, ids = env
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    poses = synth.random_poses(16 * sms + 1, ctx.ntors[ids[i]], -3.0, 3.0, seed=i)
    ref_e, ref_p, _ = ctx.local_opt(ids[i], poses, 6)
    for n in (1, 7 * sms, 7 * sms + 1, 16 * sms):
        e, p, _ = ctx.local_opt(ids[i], poses[:n], 6)
        assert np.array_equal(e, ref_e[:n]) and np.array_equal(p, ref_p[:n]), n
