"""The L-BFGS vector kernels at the sizes where they can go wrong -- fewer
entries than a warp, one CTA's last and the grid's first size (3584 entries),
histories that wrap, the general kernels' history of 9 -- against the same
iteration written with numpy on the library's own r(u) and H0 v; and a batch's,
whose members are cut into chunks of 512 entries."""
import numpy as np
import pytest

from efem_b200 import api, meshgen as mg

pytestmark = pytest.mark.gpu
ITERS = 9


def case(n, load):
    m = mg.box_hex8(0.01 * n[0], 0.01 * n[1], 0.01 * n[2], *n)
    fix = mg.nodes_where(m, lambda X: np.abs(X[:, 0]) < 1e-9)
    end = mg.nodes_where(m, lambda X: np.abs(X[:, 0] - 0.01 * n[0]) < 1e-9)
    return mg.Case(m, [mg.mat_nh()], fix, force=[([0.0, 0.0, load], end)])


def options(hist):
    o = api.default_options()
    o.m = hist
    o.max_iterations = ITERS
    o.residual_criterion = 1e-30
    return o


def lbfgs(m, o):
    """LBFGSSolver::solve with LBFGSMat and LineSearchFEA; returns x and the residual evaluations"""
    x, S, Y = np.zeros(m.n_dof), [], []
    r = m.residual(x)
    d, evals = -m.precond_apply(r), 1
    for _ in range(ITERS):
        xp, rp, dg0, step = x, r, r @ d, 1.0
        for t in range(o.max_linesearch):
            x = xp + step * d
            r = m.residual(x)
            evals += 1
            if abs(r @ d) <= abs(dg0):
                break
            step *= 1.5 if (r @ d) * dg0 > 0 else 0.5
        S, Y = (S + [x - xp])[-o.m:], (Y + [r - rp])[-o.m:]
        q, al = -r, []
        for s, y in zip(S[::-1], Y[::-1]):
            al.append((s @ q) / (s @ y))
            q = q - al[-1] * y
        d = m.precond_apply(q)
        for s, y, a in zip(S, Y, al[::-1]):
            d = d + (a - (y @ d) / (s @ y)) * s
    return x, evals


# 12, 24, 3570, 3588, 4056, 4092, 4104 and 17 424 DOFs; the load of -10 takes further line-search trials
@pytest.mark.parametrize("n,load", [((1, 1, 1), -2e-3), ((2, 1, 1), -10.0), ((14, 16, 4), -2e-3),
                                    ((13, 22, 3), -2e-3), ((8, 12, 12), -2e-3), ((341, 1, 1), -2e-3),
                                    ((8, 18, 8), -2e-3), ((24, 21, 10), -10.0)])
@pytest.mark.parametrize("hist", [1, 3, 8, 9])
def test_iterations_match_numpy(n, load, hist):
    o = options(hist)
    m = api.Model.from_case(case(n, load), o)
    u, info = m.solve()
    ref, evals = lbfgs(m, o)
    assert info["niter"] == ITERS and info["n_residual_evals"] == evals and (evals > ITERS + 1) == (load == -10.0)
    # both sides round alike but for the order of sums: eps times the condition (up to 1e6 on the slender bar)
    assert np.linalg.norm(u - ref) <= 1e-9 * np.linalg.norm(ref)


# 12, 510 and 513 (one chunk and two), 1020 and 1026 (two and three) DOFs; some
# members take further line-search trials while the others wait
@pytest.mark.parametrize("hist", [1, 3, 8])
def test_batch_iterations_match_numpy(hist):
    members = [((1, 1, 1), -2e-3), ((17, 4, 1), -2e-3), ((19, 2, 2), -2e-3), ((2, 1, 1), -10.0), ((34, 4, 1), -2e-3),
               ((38, 2, 2), -2e-3), ((8, 4, 4), -10.0)]
    o = options(hist)
    ms = [api.Model.from_case(case(n, load), o) for n, load in members]
    assert [m.n_dof for m in ms] == [12, 510, 513, 24, 1020, 1026, 600]
    us, infos = api.batch_solve(ms)
    trials = set()
    for m, u, info, (n, _) in zip(ms, us, infos, members):
        assert info["flags"] & api.SOLVE_BATCHED
        ref, evals = lbfgs(m, o)
        assert info["niter"] == ITERS and info["n_residual_evals"] == evals, n
        # the members lie apart in the union, so their J0 round to about 1e-14 instead of 1e-16
        assert np.linalg.norm(u - ref) <= 1e-8 * np.linalg.norm(ref), n
        trials.add(evals > ITERS + 1)
    assert trials == {False, True}
