"""New weights refused for want of device memory change nothing: tables, energies and scores stay
those of the weights before, and the tables can be read without device memory to spare."""
import numpy as np
import pytest

from conftest import has_gpu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("device", [False, True])
def test_refused_weights(device):
    if not has_gpu():
        pytest.skip("needs a CUDA device")
    import vdock
    from vdock import synth
    first = np.array(vdock.DEFAULT_WEIGHTS)
    second = first * [1.2, 0.8, 1.1, 0.9, 1.3, 1.4]
    ctx = vdock.Context()
    ctx.set_receptor(*synth.receptor(1000, 30.0, 1))
    ctx.set_box([0.0, 0.0, 0.0], [18.0] * 3)
    ctx.set_scoring(first, device=device)
    ctx.build_grids(list(range(17)))
    lig = ctx.add_ligand(synth.ligand(24, 5, 1))
    poses = synth.random_poses(8, 5, -3.0, 3.0, seed=1)
    want = [*ctx.tables(), ctx.energy(lig, poses), *ctx.score(lig, poses)]
    # docking more chains than fit gives up the scratch, so the next tables have no room either
    ctx.set_memory_cap(ctx.stats()["device_bytes"])
    with pytest.raises(RuntimeError, match="error 6"):
        ctx.mc_chains(lig, vdock.search_params(seed=1, n_chains=400000, search_depth=-1))
    ctx.set_memory_cap(1)
    with pytest.raises(RuntimeError, match="error 6"):
        ctx.set_scoring(second, device=True)
    tables = ctx.tables()
    ctx.set_memory_cap(0)
    got = [*tables, ctx.energy(lig, poses), *ctx.score(lig, poses)]
    for a, b in zip(got, want):
        assert np.array_equal(a, b)
    assert np.array_equal(ctx.tables()[1], want[1])
    assert np.array_equal(ctx.energy(lig, poses), want[3])
