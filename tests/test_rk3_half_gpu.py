"""The FP64 stage kernel (a thread per element and half) and the device element
order: ragged tiles, meshes whose blocks mix element kinds, instances that share
a block, both boundary fluxes, against the CPU restatement and against the
table-product kernel of the same library."""
import numpy as np
import pytest

from gdon3d_b200 import capi, kuhn
from oracle import port

pytestmark = pytest.mark.gpu

TOL = 1e-13  # FP64 rounding (2^-53) of 12 steps x 3 stages on O(1) data, with room for the growth of 1e2


def _kw(seed):
    k, kmag, p = kuhn.random_plane_wave(seed, 7.0)
    return dict(khat=k, kmag=kmag, pol=p, phase=0.3)


def _shuffled(n, seed):
    """A Kuhn mesh with its elements and vertices renumbered at random."""
    c, e = kuhn.kuhn_cube(n, 0.1, seed=seed)
    r = np.random.default_rng(seed)
    vp = r.permutation(len(c))
    cc = np.empty_like(c)
    cc[vp] = c
    return cc, vp[e][r.permutation(len(e))].astype(np.int32)


def _mesh(n, shuffle):
    return capi.mesh_build(*(_shuffled(n, n) if shuffle else kuhn.kuhn_cube(n, 0.12, seed=n)))


@pytest.mark.parametrize("n", [1, 2, 3, 5, 8])
@pytest.mark.parametrize("variant", [1, 2])
@pytest.mark.parametrize("shuffle", [False, True])
def test_fp64_stage_matches_the_oracle(n, variant, shuffle):
    mesh = _mesh(n, shuffle)
    dt = 0.3 * mesh.hmin()
    arrays = dict(face2elem=mesh.face2elem, fnode2enode=mesh.fnode2enode, boundaryface=mesh.boundaryface,
                  elem2qnode=mesh.elem2qnode, node=mesh.node)
    o = port.Oracle(mesh.nbelems, arrays, capi.tables_as_numpy(capi.t10_tables()))
    want, _ = o.rk3(port.Oracle.data(**_kw(n)), dt, 12)
    s = capi.Solver(mesh, data=capi.plane_data(**_kw(n)), dt=dt, rk3_variant=variant)
    got, _, _ = s.solve(12)
    s.close()
    assert np.linalg.norm(got - want) <= TOL * np.linalg.norm(want)


@pytest.mark.parametrize("n,shuffle", [(2, False), (5, True)])
@pytest.mark.parametrize("variant", [1, 2])
def test_fp64_metal_flux_matches_the_table_products(n, shuffle, variant):
    mesh = _mesh(n, shuffle)
    t = capi.t10_tables()
    d = 1e-13 * 600.0  # below the tolerance, above the attach check of the symmetry
    t.inv_mass[0][1] += d
    t.inv_mass[1][0] += d
    out = []
    for tabs in (None, t):
        s = capi.Solver(mesh, data=capi.plane_data(**_kw(n)), dt=0.3 * mesh.hmin(), tables=tabs, rk3_variant=variant,
                        boundary_flux=capi.BC_METAL)
        out.append(s.solve(12)[0])
        s.close()
    assert np.linalg.norm(out[0] - out[1]) <= 1e-12 * np.linalg.norm(out[1])


@pytest.mark.parametrize("precision", [capi.FP64, capi.FP32])
def test_state_norm_and_batch_follow_the_order(precision):
    """Instances of 6 to 750 elements share order blocks; states come back where
    they were put, and equal the instances alone."""
    meshes = [_mesh(n, n == 5) for n in (1, 3, 2, 5)]
    dts = [0.2 * m.hmin() for m in meshes]
    datas = [capi.plane_data(**_kw(i)) for i in range(4)]
    b = capi.BatchSolver(meshes, datas, dts, precision=precision)
    r = np.random.default_rng(3).standard_normal(b.wlen).astype(np.float32).astype(np.float64)
    b.set_state(r, 0.0)
    for (m, put, got) in zip(meshes, b.split(r), b.split(b.get_state())):
        assert np.array_equal(got[:60 * m.nbelems], put[:60 * m.nbelems])
    parts = b.split(b.solve(7)[0])
    errs = b.error_l2_batch()
    b.close()
    for m, d, dt, got, err in zip(meshes, datas, dts, parts, errs):
        s = capi.Solver(m, data=d, dt=dt, precision=precision)
        want = s.solve(7)[0]
        assert np.array_equal(got, want)
        assert abs(s.error_l2() - err) <= 1e-12 * err
        s.close()
