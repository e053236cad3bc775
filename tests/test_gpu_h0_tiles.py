"""H0 v at the sizes where the triangular solve's tiles can go wrong: fronts
of one to a few rows (pad rows, idle lanes), odd row and column counts, tiles
that hold both own and below rows, and vectors longer than one shared-memory
chunk.  L (H0 v) = v with the library's own L on the host, in the order of
rounding of L's conditioning; the application is bitwise repeatable."""
import numpy as np
import pytest

from efem_b200 import api, meshgen as mg
from test_gpu_precond_large import l_times

pytestmark = pytest.mark.gpu


def box(etype, n):
    base = mg.box_hex8(0.01 * n[0], 0.01 * n[1], 0.01 * n[2], *n)
    m = {"C3D4": lambda: mg.hex8_to_tet4(base), "C3D8": lambda: base, "C3D20": lambda: mg.hex8_to_hex20(base),
         "C3D10": lambda: mg.tet4_to_tet10(mg.hex8_to_tet4(base))}[etype]()
    fix = mg.nodes_where(m, lambda X: np.abs(X[:, 0]) < 1e-9)
    end = mg.nodes_where(m, lambda X: np.abs(X[:, 0] - 0.01 * n[0]) < 1e-9)
    return mg.Case(m, [mg.mat_nh()], fix, force=[([0.0, 0.0, -1e-3], end)])


# (18, 18, 18) C3D20: fronts of more than 1024 columns, some with rows below
@pytest.mark.parametrize("etype,n", [("C3D8", (1, 1, 1)), ("C3D4", (2, 1, 1)), ("C3D8", (3, 2, 2)), ("C3D10", (2, 1, 1)),
                                     ("C3D20", (3, 2, 1)), ("C3D8", (7, 5, 3)), ("C3D4", (13, 6, 5)), ("C3D10", (9, 4, 3)),
                                     ("C3D20", (11, 7, 5)), ("C3D8", (33, 2, 2)), ("C3D8", (2, 29, 27)), ("C3D20", (18, 18, 18))])
def test_h0_inverts_l(etype, n):
    m = api.Model.from_case(box(etype, n))
    v = np.random.default_rng(3).standard_normal(m.n_dof)
    hv = m.precond_apply(v)
    # |L| |H0| eps stays below 1e-10 on these meshes (condition numbers up to about 1e5)
    assert np.linalg.norm(l_times(m, hv) - v) <= 1e-9 * np.linalg.norm(v)
    assert np.array_equal(hv, m.precond_apply(v))
