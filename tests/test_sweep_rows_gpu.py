"""The row-driven sweeps mark values that are not written yet with a NaN pattern.
States that hold NaNs (that very pattern among them), infinities and numbers at
the ends of the range go through every sweep mode alike, and no wait gives up."""
import numpy as np
import pytest

from gdon3d_b200 import capi, kuhn

pytestmark = pytest.mark.gpu

BITS = [0xffffffffffffffff, 0xffffffff00000000, 0xfff8000000000000, 0x7ff8000000000001, 0xffffffffe0000000]


def _odd_state(n, seed):
    r = np.random.default_rng(seed)
    w = r.standard_normal(n)
    k = r.permutation(n)[:24]
    w[k[:5]] = np.array(BITS, np.uint64).view(np.float64)
    w[k[5:9]] = [np.inf, -np.inf, np.inf, -np.inf]
    w[k[9:16]] = [1e300, -1e300, 1e-300, 5e-324, 3e38, -3e38, 1e-45]
    return w


@pytest.mark.parametrize("n,nb_v", [(2, 4), (4, 6), (6, 4)])
@pytest.mark.parametrize("precision", [capi.FP64, capi.FP32, capi.FP32_REFINE, capi.BF16_STORE])
def test_odd_values_pass_through_every_mode(n, nb_v, precision):
    c, e = kuhn.kuhn_cube(n, 0.1, seed=n)
    mesh = capi.mesh_build(c, e)
    first = None
    for mode in (1, 2, 3, 4):
        s = capi.Solver(mesh, capi.SCHEME_KINETIC, capi.plane_data(), 6 * mesh.hmin(), nb_v=nb_v, precision=precision,
                        kin_sweep=mode)
        s.set_state(_odd_state(s.wlen, n), 0.0)
        s.advance(1)
        got = s.get_state()
        s.close()
        if first is None:
            first = got
            assert np.isnan(got).any() and np.isfinite(got).any()
        assert np.array_equal(got, first, equal_nan=True), mode


@pytest.mark.parametrize("precision", [capi.FP64, capi.FP32, capi.FP32_REFINE, capi.BF16_STORE])
@pytest.mark.parametrize("data", [capi.plane_data(), capi.cavity_data()])
def test_boundary_data_may_be_the_mark_itself(precision, data):
    """A time that is the NaN pattern makes boundary values that are; nothing may
    wait for them to be written."""
    c, e = kuhn.kuhn_cube(2, 0.1, seed=1)
    mesh = capi.mesh_build(c, e)
    t = np.array([BITS[0]], np.uint64).view(np.float64)[0]
    first = None
    for mode in (1, 2, 3, 4):
        s = capi.Solver(mesh, capi.SCHEME_KINETIC, data, 6 * mesh.hmin(), precision=precision, kin_sweep=mode)
        s.set_wait_limit(1 << 18)
        s.set_state(np.random.default_rng(1).standard_normal(s.wlen), t)
        s.advance(1)
        got = s.get_state()
        s.close()
        first = got if first is None else first
        assert np.array_equal(got, first, equal_nan=True), mode
