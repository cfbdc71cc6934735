"""The FP32 stage kernel holds a whole element per thread: tiles that end inside
a warp and CTAs that end inside a tile group, both register variants, both
boundary fluxes and a batch, against the FP64 path of the same library (which
the oracle pins)."""
import numpy as np
import pytest

from gdon3d_b200 import capi, kuhn

pytestmark = pytest.mark.gpu

# 12 steps x 3 stages of FP32 rounding (2^-24) on O(1) data, some tens of
# roundings per stage that add up at random
TOL = 1.5e-6


def _wave(seed):
    k, kmag, p = kuhn.random_plane_wave(seed, 7.0)
    return capi.plane_data(khat=k, kmag=kmag, pol=p, phase=0.3)


# 6, 48, 162, 384, 750, 3072 elements: 1, 2, 6, 12, 24 and 96 tiles, ragged or not
@pytest.mark.parametrize("n", [1, 2, 3, 4, 5, 8])
@pytest.mark.parametrize("variant", [1, 2])
@pytest.mark.parametrize("bc", [capi.BC_UPWIND, capi.BC_METAL])
def test_fp32_stage_matches_fp64(n, variant, bc):
    mesh = capi.mesh_build(*kuhn.kuhn_cube(n, 0.12, seed=n))
    dt = 0.3 * mesh.hmin()
    out = []
    for precision in (capi.FP64, capi.FP32):
        s = capi.Solver(mesh, data=_wave(n), dt=dt, precision=precision, rk3_variant=variant, boundary_flux=bc)
        out.append(s.solve(12)[0])
        s.close()
    assert np.linalg.norm(out[1] - out[0]) <= TOL * np.linalg.norm(out[0])


def test_fp32_batch_equals_the_instances_alone():
    meshes = [capi.mesh_build(*kuhn.kuhn_cube(n, 0.1, seed=n)) for n in (1, 3, 2, 5)]
    dts = [0.2 * m.hmin() for m in meshes]
    datas = [_wave(i) for i in range(4)]
    b = capi.BatchSolver(meshes, datas, dts, precision=capi.FP32)
    parts = b.split(b.solve(9)[0])
    b.close()
    for m, d, dt, got in zip(meshes, datas, dts, parts):
        s = capi.Solver(m, data=d, dt=dt, precision=capi.FP32)
        want = s.solve(9)[0]
        s.close()
        assert np.array_equal(got, want)


def test_fp32_state_round_trip():
    mesh = capi.mesh_build(*kuhn.kuhn_cube(3, 0.1, seed=2))
    s = capi.Solver(mesh, data=_wave(1), dt=1e-3, precision=capi.FP32)
    w = np.random.default_rng(1).standard_normal(s.wlen).astype(np.float32).astype(np.float64)
    s.set_state(w, 0.0)
    back = s.get_state()
    s.close()
    assert np.array_equal(back[:60 * mesh.nbelems], w[:60 * mesh.nbelems])


@pytest.mark.parametrize("variant", [1, 2])
@pytest.mark.parametrize("dense", [False, True])
@pytest.mark.parametrize("bc", [capi.BC_UPWIND, capi.BC_METAL])
def test_fp32_table_products_match_fp64(variant, dense, bc):
    """Tables without the P2 symmetry (a perturbed entry) keep the table-product
    kernel, which reads the same pair layout."""
    mesh = capi.mesh_build(*kuhn.kuhn_cube(3, 0.1, seed=4))
    t = capi.tables_as_numpy(capi.t10_tables())
    t["internal"][1][0][0] += 1e-6
    if dense:
        t["internal"][9][9][0] += 1e-6  # a structural zero
    tabs = capi.tables_from_numpy(t)
    out = []
    for precision in (capi.FP64, capi.FP32):
        s = capi.Solver(mesh, data=_wave(3), dt=0.3 * mesh.hmin(), precision=precision, rk3_variant=variant, tables=tabs,
                        boundary_flux=bc)
        out.append(s.solve(12)[0])
        s.close()
    assert np.linalg.norm(out[1] - out[0]) <= TOL * np.linalg.norm(out[0])
