"""The register budget where a chain's shared memory is large: 128 registers
once 80 registers' resident chains would take most of the SM's memory, in both
searches and whatever the number of chains; the chains are those of a pinned
shape."""
import numpy as np
import pytest

from conftest import has_gpu

pytestmark = pytest.mark.gpu


# (atoms, torsions), dense search, chains, shape of the first calls (4 = 80 registers, 5 = 128)
@pytest.mark.parametrize("size,dense,chains,want", [
    ((60, 15), 0, 8192, 4),    # 107 KB of 228
    ((60, 15), 1, 8192, 4),    # 158 KB
    ((66, 16), 1, 8192, 5),    # 170 KB
    ((88, 40), 0, 8192, 5),    # 194 KB
    ((88, 40), 0, 4000, 5),    # where smaller ligands explore both
    ((70, 48), 1, 8192, 5),    # two blocks per SM at any budget
    ((24, 4), 1, 8192, 4),
])
def test_large_chains(size, dense, chains, want):
    if not has_gpu():
        pytest.skip("needs a CUDA device")
    import vdock
    from vdock import synth
    ctx = vdock.Context()
    ctx.set_receptor(*synth.receptor(1200, 30.0, 2))
    ctx.set_box([0.0, 0.0, 0.0], [20.0] * 3)
    ctx.build_grids(list(range(17)))
    lig = ctx.add_ligand(synth.ligand(*size, 1))

    def dock(shape):
        r = ctx.dock_batched([lig], vdock.search_params(seed=3, n_chains=chains, search_depth=1, max_bfgs_steps=4, refine=0,
                                                        dense_bfgs=dense, launch_shape=shape))
        return r[0], ctx.stats()["dock_shape"]

    pinned, _ = dock(1)
    for _ in range(3):
        r, shape = dock(0)
        assert shape == want
        assert np.array_equal(r["energy"], pinned["energy"]) and np.array_equal(r["pose"], pinned["pose"])
        assert r["bfgs_evals"] == pinned["bfgs_evals"]
