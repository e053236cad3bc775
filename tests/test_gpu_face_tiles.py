"""Pressure faces in tiles of the element launch: face counts around the tile
sizes of every element kind and CTA size, follower and directed loads, against
the oracle (FP64, 1e-12 relative), and faces whose parent elements have no
material (their own launch)."""
import numpy as np
import pytest

import oracle
from efem_b200 import api, meshgen as mg

pytestmark = pytest.mark.gpu


def displaced(case):
    """A displacement of about 1 % strain on the free nodes."""
    free = np.setdiff1d(np.arange(case.mesh.X.shape[0]), case.fix)
    X = case.mesh.X[free]
    rng = np.random.default_rng(5)
    return (0.01 * X @ rng.uniform(-1, 1, (3, 3)) + 1e-5 * rng.normal(size=X.shape)).ravel()


@pytest.mark.parametrize("etype,n", [("C3D4", (2, 1, 1)), ("C3D4", (1, 4, 4)), ("C3D4", (1, 3, 11)), ("C3D8", (2, 1, 1)),
                                     ("C3D8", (1, 4, 4)), ("C3D8", (1, 3, 11)), ("C3D10", (2, 1, 1)), ("C3D10", (1, 2, 4)),
                                     ("C3D10", (1, 3, 3)), ("C3D20", (2, 1, 1)), ("C3D20", (1, 2, 4)), ("C3D20", (1, 3, 3))])
@pytest.mark.parametrize("load", ["pressure", "dpressure"])
def test_residual_with_faces(etype, n, load, tmp_path):
    case = mg.small_case(etype, "nh", load, n=n, size=tuple(0.01 * k for k in n))
    cfg = case.write(str(tmp_path))
    ref_model = oracle.Oracle(oracle.read_case(cfg))
    u = displaced(case)
    ref = ref_model.residual(u)
    for threads in (64, 128, 256):
        m = api.Model.from_json(cfg)
        m.set_options(elem_threads=threads)
        r = m.residual(u)
        assert np.linalg.norm(r - ref) <= 1e-12 * np.linalg.norm(ref), threads


@pytest.mark.parametrize("etype,n", [("C3D4", (1, 4, 4)), ("C3D4", (1, 3, 11)), ("C3D8", (1, 3, 11)), ("C3D10", (1, 2, 4)),
                                     ("C3D10", (1, 3, 3)), ("C3D20", (2, 1, 1)), ("C3D20", (1, 3, 3))])
@pytest.mark.parametrize("law", ["nh", "mr", "yeoh"])
@pytest.mark.parametrize("load", ["pressure", "dpressure"])
def test_tangent_with_faces(etype, n, law, load):
    check_tangent(mg.small_case(etype, law, load, n=n, size=tuple(0.01 * k for k in n)))


@pytest.mark.parametrize("etype,n", [("C3D4", (2, 2, 3)), ("C3D8", (3, 3, 3)), ("C3D10", (2, 2, 2)), ("C3D20", (3, 2, 2))])
@pytest.mark.parametrize("load", ["pressure", "dpressure", "force"])
def test_tangent_of_mixed_laws(etype, n, load):
    """Three laws in one element block: the law is chosen at run time."""
    case = mg.small_case(etype, "nh", load, n=n, size=tuple(0.01 * k for k in n))
    case.materials = [mg.mat_nh(), mg.mat_mr(C10=57000.0, C01=57000.0), mg.mat_yeoh(C10=114000.0, C20=16000.0, C30=16000.0)]
    for i, mat in enumerate(case.materials):
        mat["id"] = i + 1
    case.mesh.mat = 1 + np.arange(case.mesh.conn.shape[0]) % 3
    check_tangent(case)


def check_tangent(case):
    """K(u) v against central differences of R (truncation h^2 with h |v| about
    1e-8 m on 1e-2 m elements, cancellation eps |R| / h: 1e-6 relative holds
    both), and w.(K v) = (K^T w).v to rounding."""
    m = api.Model.from_case(case)
    u = displaced(case)
    rng = np.random.default_rng(11)
    v, w = rng.normal(size=u.size), rng.normal(size=u.size)
    kv, ktw = m.hvp(u, v), m.hvp(u, w, transpose=True)
    h = 1e-8
    fd = (m.residual(u + h * v) - m.residual(u - h * v)) / (2 * h)
    assert np.linalg.norm(kv - fd) <= 1e-6 * np.linalg.norm(kv)
    assert abs(float(w @ kv) - float(ktw @ v)) <= 1e-12 * np.linalg.norm(kv) * np.linalg.norm(w)


def test_faces_of_elements_without_a_material():
    """Two separate hexahedra, the loaded one without a material: its faces
    have no element launch to go with (the other block holds tetrahedra)."""
    X = np.array([[x, y, z] for z in (0, 1) for y in (0, 1) for x in (0, 1)], float) * 0.01
    X = np.concatenate([X, X[[0, 1, 2, 4]] + [0.1, 0, 0]])
    hexa = np.array([[0, 1, 3, 2, 4, 5, 7, 6]])
    tet = np.array([[8, 9, 10, 11]])
    blocks = [(hexa, np.array([7])), (tet, np.array([-1]))]
    m = api.Model.from_arrays(X, blocks, [{"type": "neo_hookean", "C10": 1e5, "D1": 1e-6}],
                              [("fix", np.array([8])), ("pressure", [(1, 3, 7, 5)], 1e4)])
    r = m.residual(np.zeros(m.n_dof))
    # at u = 0 the face's resultant is p A along the outward normal's opposite, R = -f
    assert np.allclose(r.reshape(-1, 3).sum(axis=0), [1e4 * 1e-4, 0, 0], rtol=1e-12, atol=1e-15)
