"""The transport sweeps take five items per warp: every sweep mode and storage
precision against the CPU restatement of the CFL-less step, on meshes whose
levels are smaller than a warp's items, end in a ragged warp or CTA, and take
several rounds of a launch's CTAs."""
import numpy as np
import pytest

from gdon3d_b200 import capi, kuhn
from oracle import port

pytestmark = pytest.mark.gpu

# relative L2 after 3 steps: FP64 rounding over the substitution chains; FP32
# and the correction's residual a few hundred units of 2^-24 and (2^-24)^2 along
# chains of up to ~80 items; BF16 storage 2^-9 per step
TOL = {capi.FP64: 1e-12, capi.FP32: 2e-5, capi.FP32_REFINE: 1e-10, capi.BF16_STORE: 2e-2}


@pytest.mark.parametrize("n,nb_v", [(1, 4), (2, 6), (3, 4), (5, 6), (7, 4)])
@pytest.mark.parametrize("precision", sorted(TOL))
def test_every_sweep_mode_matches_the_oracle(n, nb_v, precision):
    c, e = kuhn.kuhn_cube(n, 0.1, seed=n)
    mesh = capi.mesh_build(c, e)
    dt = 6 * mesh.hmin()
    k = np.array([2.0, -1.0, 2.0]) / 3.0
    kw = dict(khat=k, kmag=5.0, pol=np.array([1.0, 2.0, 0.0]) / np.sqrt(5.0), phase=0.4)
    arrays = dict(face2elem=mesh.face2elem, fnode2enode=mesh.fnode2enode, boundaryface=mesh.boundaryface,
                  elem2qnode=mesh.elem2qnode, node=mesh.node)
    o = port.Oracle(mesh.nbelems, arrays, capi.tables_as_numpy(capi.t10_tables()))
    want, _ = o.kinetic(port.Oracle.data(**kw), dt, 3, nb_v)
    first = None
    for mode in (1, 2, 3, 4):
        s = capi.Solver(mesh, capi.SCHEME_KINETIC, capi.plane_data(**kw), dt, nb_v=nb_v, precision=precision,
                        kin_sweep=mode)
        got, _, _ = s.solve(3)
        s.close()
        rel = np.linalg.norm(got - want) / np.linalg.norm(want)
        assert rel <= TOL[precision], (mode, rel)
        first = got if first is None else first
        assert np.array_equal(got, first), mode
