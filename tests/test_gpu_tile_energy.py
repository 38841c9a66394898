"""Energies of pose tiles against FP64: no further than a warp's."""
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
        o.set_box([0.0, 0.0, 0.0], [36.0] * 3)
        o.build_grids(list(range(17)))
    return ctx, orc, synth, torch.cuda.get_device_properties(0).multi_processor_count


def test_tile_energies_are_no_further_from_fp64(env):
    """Root-mean-square error against the oracle over 4 ligands' 9,475 poses each: in tiles no larger than in warps."""
    ctx, orc, synth, sms = env
    n = 64 * sms + 3
    tile = warp = 0.0
    for seed in range(4):
        lig = synth.ligand(24, 5, 100 + seed)
        lc, lo = ctx.add_ligand(lig), orc.add_ligand(lig)
        assert len(lig["pairs"]) < 400
        poses = synth.random_poses(n, 5, -3.0, 3.0, seed=seed)
        ref = np.array([orc.eval_deriv(lo, p)[0] for p in poses.astype(np.float64)])
        half = [poses[:n // 2], poses[n // 2:]]
        assert np.all(np.abs(ref) < 1e3)  # inside the box
        tile += np.sum((ctx.energy(lc, poses) - ref) ** 2)
        warp += np.sum((np.concatenate([ctx.energy(lc, p) for p in half]) - ref) ** 2)
    assert tile <= warp, (np.sqrt(tile / warp), np.sqrt(tile / (4 * n)))
