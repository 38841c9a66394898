"""Which register budget a docking launch takes by itself: 80 registers when
its chains fill the chip several times over, 128 when the longest chain
decides, both once in between; the chains are those of a pinned shape."""
import numpy as np
import pytest

from conftest import has_gpu

pytestmark = pytest.mark.gpu


# chains, (ligand atoms, torsions) list, shapes of the first calls; launch_shape 4 = 80 registers, 5 = 128.
# 24 chains resident per SM at 80 registers: 3,552 on 148 SMs.
@pytest.mark.parametrize("chains,sizes,first", [
    (8192, [(24, 4)], [4, 4, 4]),               # 0.43 of an even share
    (4000, [(24, 4)], [4, 5, None]),            # 0.89
    (2048, [(24, 4)], [5, 5, 5]),               # 1.73
    (1100, [(12, 2), (36, 9)], [5, 5, 5]),      # the large ligand's chains are most of the work: > 1.6
    (7200, [(12, 2), (36, 9)], [4, 4, 4]),      # < 0.5
])
def test_shape_rule(chains, sizes, first):
    if not has_gpu():
        pytest.skip("needs a CUDA device")
    import vdock
    from vdock import synth
    xyz, xs = synth.receptor(1200, 30.0, 2)
    ctx = vdock.Context()
    ctx.set_receptor(xyz, xs)
    ctx.set_box([0.0, 0.0, 0.0], [16.0] * 3)
    ctx.build_grids(synth.TYPES8)
    ligs = [ctx.add_ligand(synth.ligand(na, nt, 1)) for na, nt in sizes]

    def dock(shape):
        r = ctx.dock_batched(ligs, vdock.search_params(seed=3, n_chains=chains, search_depth=1, max_bfgs_steps=5,
                                                       refine=0, launch_shape=shape))
        return r, ctx.stats()["dock_shape"]

    pinned, _ = dock(1)
    for want in first:
        r, shape = dock(0)
        assert shape == want if want else shape in (4, 5)
        for a, b in zip(r, pinned):
            assert np.array_equal(a["energy"], b["energy"]) and np.array_equal(a["pose"], b["pose"])
            assert a["bfgs_evals"] == b["bfgs_evals"]
