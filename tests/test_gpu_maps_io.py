"""Grid build and map read-back where their host and device splits change.

Corner cells: columns of 4 cells along z (remainders 0 to 3, boxes of one and
two cells), every map group width (1 to 4, 5 to 8, 9 to 12 and 13 to 17 maps).
The cells are read through the evaluation: a one-atom pose at a cell's centre
is the mean of the cell's eight map values, in the box's far corner too.
Read-back: maps of one slab and of several, padded and unpadded rows, through
the pageable and (after 40 reads) the pinned buffer.  A rebuild that keeps its
allocations gives what a new context gives.
"""
import numpy as np
import pytest

import oracle_lib as O
from conftest import has_gpu

pytestmark = pytest.mark.gpu


def _atom(t):
    """A rigid two-atom ligand, the second atom a hydrogen (no energy)."""
    return dict(n_atoms=2, xyz=np.array([[0.0, 0, 0], [1.0, 0, 0]]), xs=np.array([t, -1], np.int32),
                el=np.array([1, 0], np.int32), atom_node=np.zeros(2, np.int32), node_parent=np.array([-1], np.int32),
                node_origin_atom=np.zeros(1, np.int32), node_axis_atom=np.array([-1], np.int32),
                pairs=np.zeros((0, 2), np.int32), num_tors=0.0)


@pytest.mark.parametrize("size,n_types", [((0.3, 0.3, 0.3), 1), ((0.7, 0.4, 1.2), 4), ((3.0, 2.6, 1.9), 5), ((6.0, 7.1, 8.3), 12),
                                          ((23.0, 9.0, 4.0), 17)])
def test_cells_are_the_maps(size, n_types):
    if not has_gpu():
        pytest.skip("needs a CUDA device")
    import vdock
    from vdock import synth
    types = list(range(17))[-n_types:]
    ctx = vdock.Context()
    ctx.set_receptor(*synth.receptor(300, 14.0, 4))
    ctx.set_box([0.1, -0.2, 0.3], size)
    ctx.build_grids(types)
    n, b, e = ctx.grid_dims()
    rng = np.random.default_rng(1)
    for t in types:
        m = ctx.grid(t).astype(np.float64)
        lig = ctx.add_ligand(_atom(t))
        cell = np.concatenate([rng.integers(0, n - 1, size=(40, 3)), [[0, 0, 0]], [n - 2]])
        poses = np.zeros((len(cell), 7), np.float32)
        poses[:, :3] = b + (cell + 0.5) * (e - b) / (n - 1)
        poses[:, 3] = 1.0
        x, y, z = cell.T
        corners = np.stack([m[z + k, y + j, x + i] for i in (0, 1) for j in (0, 1) for k in (0, 1)])
        # curl cap off: v large.  FP32: the atom is ~1e-6 A off the centre (at most
        # 8 ulp of 20 A), 5e-6 cells, and the sum rounds eight times
        got = ctx.energy(lig, poses, vdock.eval_params(v_inter=1e12))
        tol = 5e-6 * np.ptp(corners, axis=0) + 8 * 6e-8 * np.abs(corners).sum(0) + 1e-6
        assert np.all(np.abs(got - corners.mean(0)) <= tol), t


def test_map_read_back_and_rebuild():
    if not has_gpu():
        pytest.skip("needs a CUDA device")
    import vdock
    from vdock import synth
    xyz, xs = synth.receptor(600, 20.0, 4)

    def context(size, types):
        c = vdock.Context()
        c.set_receptor(xyz, xs)
        c.set_box([0.0, 0.0, 0.0], size)
        c.build_grids(types)
        return c

    # rows of 20 floats (unpadded), of 62 (padded); 33 slabs' worth in the last
    for size in ((7.0, 5.0, 6.0), (22.7, 3.0, 9.0), (40.0, 30.0, 90.0)):
        ctx, orc = context(size, [0, 3, 8]), O.Oracle()
        first = {t: ctx.grid(t) for t in (0, 3, 8)}
        if size[2] < 50:
            orc.set_receptor(xyz, xs)
            orc.set_box([0.0, 0.0, 0.0], size)
            orc.build_grids([0, 3, 8])
            for t in first:
                ref = orc.grid(t)
                assert np.max(np.abs(first[t] - ref) / np.maximum(np.abs(ref), 1.0)) <= 1e-5
        for _ in range(45):  # past the reads after which the buffer is pinned
            again = ctx.grid(3)
        assert np.array_equal(again, first[3])
        # the same size again with another receptor, then the first one: allocations kept
        ctx.set_receptor(xyz + 0.25, xs)
        ctx.build_grids([0, 3, 8])
        assert not np.array_equal(ctx.grid(0), first[0])
        held = ctx.stats()["device_bytes"]
        ctx.set_receptor(xyz, xs)
        ctx.build_grids([0, 3, 8])
        assert ctx.stats()["device_bytes"] == held
        for t in first:
            assert np.array_equal(ctx.grid(t), first[t])
