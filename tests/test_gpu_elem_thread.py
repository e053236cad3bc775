"""The FP32 kernel that sums an element's forces in registers (k_elem_thread, 20
nodes and 27 points): element counts around a warp's 32, every law and a
mixture, faces on the same launch, against the oracle."""
import numpy as np
import pytest

import oracle
from efem_b200 import api, meshgen as mg
from test_gpu_face_tiles import displaced

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [(1, 1, 1), (31, 1, 1), (4, 4, 2), (11, 3, 1), (13, 5, 1)])
@pytest.mark.parametrize("law", ["nh", "mr", "yeoh", "two"])
def test_residual_27_points_fp32(n, law, tmp_path):
    case = mg.small_case("C3D20", "nh" if law == "two" else law, "pressure", n=n, size=tuple(0.01 * k for k in n))
    if law == "two":
        case.materials = [mg.mat_nh(), mg.mat_yeoh(C10=114000.0, C20=16000.0, C30=16000.0)]
        for i, mat in enumerate(case.materials):
            mat["id"] = i + 1
        case.mesh.mat = 1 + np.arange(case.mesh.conn.shape[0]) % 2
    cfg = case.write(str(tmp_path))
    u = displaced(case)
    ref = oracle.Oracle(oracle.read_case(cfg)).residual(u)
    err = {}
    for split in (False, True):
        m = api.Model.from_json(cfg)
        m.set_options(precision=api.MIXED, elem_threads=1 if split else 128)
        err[split] = np.linalg.norm(m.residual(u) - ref) / np.linalg.norm(ref)
        if split:
            assert m.info()["elem_threads_fp32"] == 64
    # the same products and sums in FP32, added up in another order: not less accurate than the other kernel
    assert err[True] <= 1.5 * err[False] + 1e-7, err


def test_the_option_forces_the_kernel(tmp_path):
    """elem_threads = 1 takes it without timing, in deterministic mode too; the
    FP64 kernel, which has no such variant, stays at what that mode fixes."""
    cfg = mg.small_case("C3D20", "nh", "pressure", n=(2, 1, 1)).write(str(tmp_path))
    m = api.Model.from_json(cfg)
    u = np.zeros(m.n_dof)
    for threads, want in ((1, 64), (0, 128)):
        m.set_options(precision=api.MIXED, deterministic=1, elem_threads=threads)
        m.residual(u)
        assert m.info()["elem_threads_fp32"] == want and m.info()["elem_threads_fp64"] == 128
