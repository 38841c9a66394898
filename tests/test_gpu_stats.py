"""vd_stats: what a call adds does not depend on what the context did before, and
the corner cells' time is the kernel's."""
import pytest

from conftest import has_gpu

pytestmark = pytest.mark.gpu


@pytest.fixture()
def vd():
    if not has_gpu():
        pytest.skip("needs a CUDA device")
    import vdock
    return vdock


def test_evaluation_counts(vd):
    from vdock import synth
    ctx = vd.Context()
    ctx.set_receptor(*synth.receptor(1000, 30.0, 1))
    ctx.set_box([0.0, 0.0, 0.0], [18.0] * 3)
    ctx.build_grids(synth.TYPES8)
    lig = ctx.add_ligand(synth.ligand(20, 4, 1))
    poses = synth.random_poses(6, 4, -3.0, 3.0, seed=1)
    sp = vd.search_params(seed=1, n_chains=64, search_depth=2, refine=1)
    bare = vd.search_params(seed=1, n_chains=64, search_depth=2, refine=0)

    def counted(call):
        before = ctx.stats()["bfgs_evals"]
        out = call()
        return ctx.stats()["bfgs_evals"] - before, out

    dock, r = counted(lambda: ctx.dock_batched([lig], sp))
    assert dock > r[0]["bfgs_evals"] > 0  # the search's and the refinement's
    refine, _ = counted(lambda: ctx.refine(lig, poses))
    assert refine >= len(poses)
    for _ in range(2):
        assert counted(lambda: ctx.dock_batched([lig], sp))[0] == dock
        assert counted(lambda: ctx.dock_plain(lig, sp))[0] == dock
        assert counted(lambda: ctx.refine(lig, poses))[0] == refine
        n, out = counted(lambda: ctx.dock_batched([lig], bare))
        assert n == out[0]["bfgs_evals"] == r[0]["bfgs_evals"]
        n, (_, _, ev) = counted(lambda: ctx.mc_chains(lig, bare))
        assert n == ev == r[0]["bfgs_evals"]
        n, (_, _, ev) = counted(lambda: ctx.local_opt(lig, poses, 5))
        assert n == ev
        assert counted(lambda: ctx.energy_grad(lig, poses))[0] == len(poses)


def test_cell_time_is_the_kernels(vd):
    """A build that allocates the cells against one that keeps them: the same kernel on the same sizes (1.1 GB written,
    about 0.2 ms); the bound leaves half of that for clocks."""
    from vdock import synth
    ctx = vd.Context()
    ctx.set_receptor(*synth.receptor(1000, 30.0, 1))
    ctx.set_box([0.0, 0.0, 0.0], [12.0] * 3)
    ctx.build_grids(synth.TYPES8)  # loads the kernels
    ctx.set_box([0.0, 0.0, 0.0], [60.0] * 3)
    ctx.build_grids(synth.TYPES8)
    first = ctx.stats()["cells_ms"]
    again = []
    for _ in range(3):
        ctx.build_grids(synth.TYPES8)
        again.append(ctx.stats()["cells_ms"])
    assert 0 < first <= 1.5 * max(again), (first, again)
