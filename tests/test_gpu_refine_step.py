"""One refinement step from optimised starts: every returned energy is its pose's direct-sum energy and none is above its
start's, also where the line search stops at another step than the oracle's."""
import numpy as np
import pytest

import oracle_lib as O
from conftest import has_gpu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rec_atoms,radius,na,nt", [(2000, 40.0, 5, 1), (1200, 24.0, 33, 9), (2000, 40.0, 65, 15),
                                                    (2000, 40.0, 100, 20)])
def test_one_step(rec_atoms, radius, na, nt):
    if not has_gpu():
        pytest.skip("needs a CUDA device")
    import vdock
    from vdock import synth
    xyz, xs = synth.receptor(rec_atoms, radius, 9)
    lig = synth.ligand(na, nt, 5)
    ctx, orc = vdock.Context(), O.Oracle()
    for o in (ctx, orc):
        o.set_receptor(xyz, xs)
        o.set_box([0.0, 0.0, 0.0], [34.0] * 3)
        o.build_grids(list(range(17)))
    lc, lo = ctx.add_ligand(lig), orc.add_ligand(lig)
    starts = synth.random_poses(21, ctx.ntors[lc], -2.0, 2.0, seed=na)
    _, starts, _ = ctx.local_opt(lc, starts, 20)
    _, b, en = orc.grid_info()
    e, p = ctx.refine(lc, starts, 1)
    checked = 0
    for i in range(len(starts)):
        x = [orc.coords(lo, q[i].astype(np.float64), lig["n_atoms"]) for q in (starts, p)]
        if not (e[i] < 1e30 and all(np.all((c > b) & (c < en)) for c in x)):
            continue
        checked += 1
        s, r = [orc.eval_deriv(lo, q[i].astype(np.float64), v=(1000, 1000, 1000), slope=1e6, noncache=True)[0]
                for q in (starts, p)]
        assert abs(r - e[i]) <= 2e-3 * max(1.0, abs(r)), (i, r, e[i])
        assert e[i] <= s + 2e-3 * max(1.0, abs(s)), (i, s, e[i])
    assert checked >= 10
