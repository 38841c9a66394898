"""A pose's energy and gradient against the number of poses beside it.  The
number picks the kernel (a team per pose, a warp per pose, tiles of 1 to 32
poses), and each adds in an order of its own: coordinates and the terms are the
same, sums may differ by their rounding.
"""
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
    ctx.set_receptor(*synth.receptor(1000, 30.0, 3))
    ctx.set_box([0.0, 0.0, 0.0], [36.0] * 3)
    ctx.build_grids(list(range(17)))
    return ctx, synth, torch.cuda.get_device_properties(0).multi_processor_count


@pytest.mark.parametrize("na,nt", [(2, 0), (12, 2), (24, 5), (40, 10), (60, 15)])
def test_sums_by_number_of_poses(env, na, nt):
    """FP32 sums of the same terms in two orders differ by at most their additions times 2^-24 of the terms' sum each: up
    to 40 additions on a term's way (a tile's slot of 25 pairs and 4 atoms, 16 warps), terms between -0.7 and 10
    (pairs) and -3 and 10 (atoms).  Gradients: a tenth of the tolerance to the oracle."""
    ctx, synth, sms = env
    lig = synth.ligand(na, nt, 5)
    lc = ctx.add_ligand(lig)
    pairs = len(lig["pairs"])
    poses = synth.random_poses(64 * sms + 3, nt, -3.0, 3.0, seed=na)
    e_all, g_all = ctx.energy_grad(lc, poses)
    for n in (1, 7 * sms, 7 * sms + 1, 3 * sms, 16 * sms + 5, 32 * sms + 7, 64 * sms - 1):
        e, g = ctx.energy_grad(lc, poses[:n])
        only = ctx.energy(lc, poses[:n])
        terms = np.abs(e) + 2 * (0.7 * pairs + 3 * na)
        for a in (e_all[:n], only):
            assert np.all(np.abs(e - a) <= 2 * 40 * 2.0 ** -24 * terms), n
        assert np.all(np.abs(g - g_all[:n]) <= 1e-4 * np.maximum(1.0, np.abs(g_all[:n]).max(1, keepdims=True))), n
