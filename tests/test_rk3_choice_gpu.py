"""FP64 RK3 has two stage kernels whose sums round differently.  Which of them a
handle runs follows from the mesh and the device, not from a timing, so that equal
calls give equal bits in every process; the FP32 kernels and those of other tables
differ in registers only."""
import numpy as np
import pytest

from gdon3d_b200 import capi, kuhn

pytestmark = pytest.mark.gpu


def _sms():
    import torch
    return torch.cuda.get_device_properties(0).multi_processor_count


def _wave(seed):
    k, kmag, p = kuhn.random_plane_wave(seed, 7.0)
    return capi.plane_data(khat=k, kmag=kmag, pol=p, phase=0.3)


def _mesh(n, shuffle=False):
    c, e = kuhn.kuhn_cube(n, 0.1, seed=n)
    if shuffle:
        e = e[np.random.default_rng(n).permutation(len(e))]
    return capi.mesh_build(c, e)


def _attach(mesh, **kw):
    s = capi.Solver(mesh, dt=1e-4, **kw)
    out = s.rk3_variant[0], s.launches
    s.close()
    return out


@pytest.mark.parametrize("n,shuffle", [(1, False), (8, False), (11, False), (12, False), (24, True), (32, True),
                                       (20, False)])
def test_fp64_kernel_is_chosen_without_timing(n, shuffle):
    """The attach launches what it launches with the kernel given, no trials."""
    mesh = _mesh(n, shuffle)
    tiles = (mesh.nbelems + 31) // 32
    import torch
    beyond_l2 = 2 * tiles * 1920 * 8 > torch.cuda.get_device_properties(0).L2_cache_size
    want = 1 if tiles <= 2 * _sms() or (shuffle and beyond_l2) else 2
    variant, launches = _attach(mesh)
    assert variant == want
    assert launches == _attach(mesh, rk3_variant=want)[1]


def test_other_tables_do_not_set_the_choice():
    """Tables that never run the half kernel, attached first at the same size."""
    mesh = _mesh(9)
    t = capi.tables_as_numpy(capi.t10_tables())
    t["internal"][1][0][0] += 1e-6
    _attach(mesh, tables=capi.tables_from_numpy(t))
    assert _attach(mesh)[0] == (1 if (mesh.nbelems + 31) // 32 <= 2 * _sms() else 2)


@pytest.mark.parametrize("precision,variant", [(capi.FP64, 1), (capi.FP64, 2), (capi.FP32, 1), (capi.FP32, 2)])
def test_batch_equals_the_instances_with_each_kernel(precision, variant):
    """Instances of 6 to 750 elements with their own time steps and data."""
    meshes = [_mesh(n, n == 5) for n in (1, 3, 2, 5)]
    dts = [0.2 * m.hmin() for m in meshes]
    datas = [_wave(i) for i in range(4)]
    b = capi.BatchSolver(meshes, datas, dts, precision=precision, rk3_variant=variant)
    parts = b.split(b.solve(7)[0])
    b.close()
    for m, d, dt, got in zip(meshes, datas, dts, parts):
        s = capi.Solver(m, data=d, dt=dt, precision=precision, rk3_variant=variant)
        want = s.solve(7)[0]
        s.close()
        assert np.array_equal(got, want)


@pytest.mark.parametrize("precision,tables", [(capi.FP32, "p2"), (capi.FP32, "other"), (capi.FP64, "other")])
@pytest.mark.parametrize("bc", [capi.BC_UPWIND, capi.BC_METAL])
def test_register_caps_give_the_same_bits(precision, tables, bc):
    """Where the faster variant is still timed, both give the same state."""
    mesh = _mesh(4)
    t = None
    if tables == "other":
        t = capi.tables_as_numpy(capi.t10_tables())
        t["internal"][1][0][0] += 1e-6
        t = capi.tables_from_numpy(t)
    out = []
    for variant in (1, 2):
        s = capi.Solver(mesh, data=_wave(2), dt=0.2 * mesh.hmin(), precision=precision, tables=t, rk3_variant=variant,
                        boundary_flux=bc)
        out.append(s.solve(9)[0])
        s.close()
    assert np.array_equal(out[0], out[1])


def _other_tables():
    t = capi.tables_as_numpy(capi.t10_tables())
    t["internal"][1][0][0] += 1e-6
    return capi.tables_from_numpy(t)


@pytest.mark.parametrize("n,shuffle", [(2, False), (10, False), (13, False), (18, False), (26, False), (26, True)])
@pytest.mark.parametrize("precision,other", [(capi.FP32, False), (capi.FP32, True), (capi.FP64, True)])
def test_no_kernel_is_chosen_by_timing(n, shuffle, precision, other):
    """FP32 takes the larger register budget with the P2 tables.  Other tables take
    it while its CTAs are resident at once and where gathers are scattered."""
    mesh = _mesh(n, shuffle)
    tiles = (mesh.nbelems + 31) // 32
    want = 1 if not other or shuffle or tiles <= (2 if precision == capi.FP64 else 4) * _sms() else 2
    kw = dict(precision=precision, tables=_other_tables() if other else None)
    variant, launches = _attach(mesh, **kw)
    assert variant == want
    assert launches == _attach(mesh, rk3_variant=want, **kw)[1]
