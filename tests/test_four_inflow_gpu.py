"""An element whose four faces all are inflow.  No conforming mesh has one (the
scaled normals of a tetrahedron add up to zero), but the attach takes meshes whose
two sides of a face are different points, and the normal of a face is its L side's:
clusters of a central element (R side) and neighbours, each turned about its own
centroid until its face looks into the centre along the first velocity."""
import numpy as np
import pytest

from gdon3d_b200 import capi
from oracle import port

LAM = capi.D3Q4_LAMBDA
V0 = LAM * np.array(capi.D3Q4_VI[0], float)
FACES = np.array([[0, 3, 2], [0, 1, 3], [0, 2, 1], [1, 2, 3]])  # outward, local vertices


def _normal(x, f):
    a, b, c = x[FACES[f]]
    return np.cross(b - a, c - a)


def _cluster(r, boundary):
    """Vertices of the central tetrahedron and the tetrahedra on its faces.
    boundary: -1, or the central face (inflow by its own normal) left without one."""
    while True:
        x = r.standard_normal((4, 3))
        if np.linalg.det(x[1:] - x[:1]) < 0:
            x[[0, 1]] = x[[1, 0]]
        if np.linalg.det(x[1:] - x[:1]) > 0.5 and (boundary < 0 or V0 @ _normal(x, boundary) < -0.2):
            break
    elems = []
    for f in range(4):
        if f == boundary:
            continue
        tri = FACES[f]
        apex = x[tri].mean(0) + _normal(x, f) * 0.8
        elems.append((tri[[0, 2, 1]], apex))
    return x, elems


def make_mesh(seed, clusters=12):
    """MeshArrays of disjoint clusters, every element with points of its own."""
    r = np.random.default_rng(seed)
    coords, tets, centre = [], [], []
    for c in range(clusters):
        x, elems = _cluster(r, c % 5 - 1)
        x = x + 10.0 * c
        base = sum(len(a) for a in coords)
        pts = [x] + [np.asarray(a)[None] + 10.0 * c for _, a in elems]
        coords.extend(pts)
        centre.append(len(tets))  # before its neighbours: the later element is a face's L side
        tets.append([base, base + 1, base + 2, base + 3])
        for k, (tri, _) in enumerate(elems):
            t = [base + tri[0], base + tri[1], base + tri[2], base + 4 + k]
            p = np.concatenate(pts)[np.array(t) - base]
            if np.linalg.det(p[1:] - p[:1]) < 0:
                t[0], t[1] = t[1], t[0]
            tets.append(t)
    m = capi.mesh_build(np.concatenate(coords), np.array(tets, np.int32))
    ne = m.nbelems
    f2e = m.face2elem.reshape(-1, 4)
    # points of its own for every element, boundary faces among them
    q = m.elem2qnode[:10 * ne].reshape(ne, 10)
    node = m.node.reshape(-1, 3)[q].reshape(ne, 10, 3).copy()
    e2q = np.arange(10 * ne).reshape(ne, 10)
    fn = m.fnode2enode.reshape(-1, 12)
    tail = [e2q[f2e[F, 0], fn[F, :6]] for F in m.boundaryface]
    # turn the neighbours whose face looks away: half a turn about an axis across V0
    axis = np.cross(V0, [0.3, -1.0, 0.5])
    axis /= np.linalg.norm(axis)
    turn = 2 * np.outer(axis, axis) - np.eye(3)
    for eL, fL, eR, _ in f2e:
        if eR in centre:
            if V0 @ _normal(node[eL, :4], fL) <= 0:
                mid = node[eL].mean(0)
                node[eL] = (node[eL] - mid) @ turn.T + mid
            assert V0 @ _normal(node[eL, :4], fL) > 0
    count = np.zeros(ne, int)
    for eL, fL, eR, fR in f2e:
        s = V0 @ _normal(node[eL, :4], fL)
        count[eL] += s < 0
        if eR >= 0:
            count[eR] += s > 0
    assert (count[centre] == 4).all()
    out = capi.MeshArrays(m.face2elem, m.fnode2enode, m.boundaryface, np.concatenate([e2q.ravel(), np.ravel(tail)]),
                          node.ravel(), ne)
    return out


def _wave():
    return dict(khat=np.array([2.0, -1.0, 2.0]) / 3.0, kmag=1.3, pol=np.array([1.0, 2.0, 0.0]) / np.sqrt(5.0), phase=0.4)


def _oracle(mesh, dt, steps):
    arrays = dict(face2elem=mesh.face2elem, fnode2enode=mesh.fnode2enode, boundaryface=mesh.boundaryface,
                  elem2qnode=mesh.elem2qnode, node=mesh.node)
    o = port.Oracle(mesh.nbelems, arrays, capi.tables_as_numpy(capi.t10_tables()))
    return o.kinetic(port.Oracle.data(**_wave()), dt, steps, 4)[0]


def test_the_oracle_solves_the_mesh():
    w = _oracle(make_mesh(3), 0.05, 2)
    assert np.isfinite(w).all() and np.linalg.norm(w) > 0


# relative L2 after 3 steps, as in the tests of ordinary meshes: FP64 rounding; FP32 and
# the correction's residual a few hundred units of 2^-24 and (2^-24)^2.  BF16 storage
# only has to give the same bits in every mode (its sweeps are the FP32 ones; what its
# rounding grows to on a mesh that does not conform has no bound to hold it against).
TOL = {capi.FP64: 1e-12, capi.FP32: 2e-5, capi.FP32_REFINE: 1e-10, capi.BF16_STORE: np.inf}


@pytest.mark.gpu
@pytest.mark.parametrize("precision", sorted(TOL))
def test_every_sweep_mode_takes_four_inflow_faces(precision):
    mesh = make_mesh(3)
    want = _oracle(mesh, 0.05, 3)
    first = None
    for mode in (1, 2, 3, 4):
        s = capi.Solver(mesh, capi.SCHEME_KINETIC, capi.plane_data(**_wave()), 0.05, precision=precision, kin_sweep=mode)
        got, _, _ = s.solve(3)
        s.close()
        rel = np.linalg.norm(got - want) / np.linalg.norm(want)
        assert rel <= TOL[precision], (mode, rel)
        first = got if first is None else first
        assert np.array_equal(got, first), mode
