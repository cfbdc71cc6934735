"""The device element order is taken where it brings the neighbours of a tile
together, and the mesh's own order elsewhere: the gmsh meshes keep theirs.  Either
way the states are the oracle's."""
import os

import numpy as np
import pytest

from gdon3d_b200 import capi, kuhn
from oracle import port

pytestmark = pytest.mark.gpu

GOLDEN = os.path.join(os.path.dirname(os.path.abspath(__file__)), "golden", "ref_meshes.npz")
TOL = 1e-13  # FP64 rounding (2^-53) of 12 steps x 3 stages on O(1) data, with room for the growth of 1e2


def _mesh(name):
    if name.startswith("kuhn"):
        return capi.mesh_build(*kuhn.kuhn_cube(int(name[4:]), 0.1, seed=1))
    z = np.load(GOLDEN)
    return capi.mesh_build(z[name + "_coords"], z[name + "_elem2node"])


def _attach_launches(name, precision):
    s = capi.Solver(_mesh(name), dt=1e-4, precision=precision, rk3_variant=1)
    n = s.launches
    s.close()
    return n


@pytest.mark.parametrize("precision", [capi.FP64, capi.FP32])
@pytest.mark.parametrize("name", ["t4_cube_16", "t4_cube_8_torus_128"])
def test_a_gmsh_mesh_keeps_its_order(name, precision):
    """Going back to the mesh's order is one launch more."""
    assert _attach_launches(name, precision) == _attach_launches("kuhn8", precision) + 1


@pytest.mark.parametrize("name", ["t4_cube_8", "kuhn1", "kuhn6"])
@pytest.mark.parametrize("variant", [1, 2])
def test_states_of_both_orders_match_the_oracle(name, variant):
    mesh = _mesh(name)
    kw = dict(khat=np.array([2.0, -1.0, 2.0]) / 3.0, kmag=5.0, pol=np.array([1.0, 2.0, 0.0]) / np.sqrt(5.0), phase=0.4)
    arrays = dict(face2elem=mesh.face2elem, fnode2enode=mesh.fnode2enode, boundaryface=mesh.boundaryface,
                  elem2qnode=mesh.elem2qnode, node=mesh.node)
    dt = 0.3 * mesh.hmin()
    want, _ = port.Oracle(mesh.nbelems, arrays, capi.tables_as_numpy(capi.t10_tables())).rk3(port.Oracle.data(**kw), dt, 12)
    s = capi.Solver(mesh, data=capi.plane_data(**kw), dt=dt, rk3_variant=variant)
    got, _, _ = s.solve(12)
    back = s.get_state()
    s.close()
    assert np.linalg.norm(got - want) <= TOL * np.linalg.norm(want)
    assert np.array_equal(back, got)
