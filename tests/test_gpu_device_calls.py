"""Evaluations in flight on a caller's stream while the context changes what
they read: they return what they would have returned alone, bit for bit.  The
stream is held back first, so the evaluations run only after the change has
been asked for unless the change waits for them.
"""
import numpy as np
import pytest

from conftest import has_gpu

pytestmark = pytest.mark.gpu

HOLD = 100_000_000  # cycles, about 50 ms


@pytest.fixture()
def env():
    if not has_gpu():
        pytest.skip("needs a CUDA device")
    import torch
    import vdock
    from vdock import synth
    xyz, xs = synth.receptor(1500, 35.0, 3)
    ctx = vdock.Context()
    ctx.set_receptor(xyz, xs)
    ctx.set_box([0.0, 0.0, 0.0], [24.0] * 3)
    ctx.build_grids(list(range(17)))
    lig = ctx.add_ligand(synth.ligand(30, 6, 2))
    return torch, vdock, synth, ctx, lig, xyz, xs


def _buffers(torch, synth, ctx, lig, n):
    p = torch.from_numpy(synth.random_poses(n, ctx.ntors[lig], -5.0, 5.0, seed=n)).cuda()
    return p, torch.empty(n, device="cuda"), torch.empty(n, p.shape[1] - 1, device="cuda")


@pytest.mark.parametrize("n", [64, 20000])
@pytest.mark.parametrize("captured", [False, True])
def test_rebuild_of_the_same_box(env, n, captured):
    torch, vd, synth, ctx, lig, xyz, xs = env
    p, e, g = _buffers(torch, synth, ctx, lig, n)

    def evaluate():
        ctx.energy_grad_device(lig, n, p.data_ptr(), e.data_ptr(), g.data_ptr(), torch.cuda.current_stream().cuda_stream)

    side = torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.stream(side):
        evaluate()
    side.synchronize()
    alone = e.clone(), g.clone()
    torch.cuda.synchronize()
    with torch.cuda.stream(side):
        if captured:
            graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(graph, stream=side):
                evaluate()
            e.zero_()
        torch.cuda._sleep(HOLD)
        graph.replay() if captured else evaluate()
    ctx.set_receptor(xyz + 0.3, xs)
    ctx.build_grids(list(range(17)))
    torch.cuda.synchronize()
    assert torch.equal(e, alone[0]) and torch.equal(g, alone[1])
    with torch.cuda.stream(side):
        evaluate()
    torch.cuda.synchronize()
    assert not torch.equal(e, alone[0])  # the new receptor's


@pytest.mark.parametrize("change", ["scoring", "scoring_device", "ligands"])
def test_new_tables_and_ligands(env, change):
    torch, vd, synth, ctx, lig, xyz, xs = env
    p, e, g = _buffers(torch, synth, ctx, lig, 20000)
    side = torch.cuda.Stream()

    def evaluate():
        ctx.energy_grad_device(lig, len(p), p.data_ptr(), e.data_ptr(), g.data_ptr(), side.cuda_stream)

    torch.cuda.synchronize()
    evaluate()
    side.synchronize()
    alone = e.clone(), g.clone()
    torch.cuda.synchronize()
    with torch.cuda.stream(side):
        torch.cuda._sleep(HOLD)
        evaluate()
    if change == "ligands":
        other = synth.ligand(30, 6, 9)
        ctx.clear_ligands()
        ctx.pose_coords(ctx.add_ligand(other), synth.random_poses(2, 6, -1.0, 1.0, seed=1))  # uploads it
    else:
        ctx.set_scoring(1.5 * np.array(vd.DEFAULT_WEIGHTS), device=change == "scoring_device")
    torch.cuda.synchronize()
    assert torch.equal(e, alone[0]) and torch.equal(g, alone[1])


def test_ligand_uploaded_under_capture(env):
    """A ligand in a cleared one's place, first used by a call that is being captured."""
    torch, vd, synth, ctx, lig, xyz, xs = env
    p, e, g = _buffers(torch, synth, ctx, lig, 64)
    side = torch.cuda.Stream()
    torch.cuda.synchronize()
    ctx.energy_grad_device(lig, 64, p.data_ptr(), e.data_ptr(), g.data_ptr(), side.cuda_stream)
    side.synchronize()
    ctx.clear_ligands()
    lig = ctx.add_ligand(synth.ligand(30, 6, 9))
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=side, capture_error_mode="relaxed"):
        ctx.energy_grad_device(lig, 64, p.data_ptr(), e.data_ptr(), g.data_ptr(), side.cuda_stream)
    graph.replay()
    torch.cuda.synchronize()
    want_e, want_g = ctx.energy_grad(lig, p.cpu().numpy())
    assert np.array_equal(e.cpu().numpy(), want_e) and np.array_equal(g.cpu().numpy(), want_g)
