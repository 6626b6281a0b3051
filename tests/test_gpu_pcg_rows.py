"""The PCG of instances without contact blocks (rows, slices and halo lists per
CTA): directions against the oracle's direct solve at the sizes where its cut
changes (one CTA, several, partial slices and rows per CTA forced down), with
fixed vertices, in both precisions; and an arena of such instances bit for bit
as alone.

Tolerances are those of the other direction tests: 1e-6 in FP64 (PCG to 1e-8
times the system's condition), 2e-3 in mixed mode (FP32 element Hessians).
"""
import numpy as np
import pytest

import cases
from test_gpu_parity import ctx_for, oracle_problem

pytestmark = pytest.mark.gpu

# grid of the bar, parameters: V = 12 (a slice and a half), 40 / 45 (largest
# single FP64 CTA and the next), 192 / 200 (largest single mixed CTA and the
# next), 963 (16 or 25 CTAs), one CTA of 320 and two of 160 rows (slices per warp),
# rows per CTA forced to 16 and to 7
FORCED = lambda rows: {"pcg_grid_min_vertices": 1, "pcg_grid_cta_vertices": rows}  # noqa: E731
SIZES = [((1, 1, 2), {}), ((1, 4, 3), {}), ((2, 2, 4), {}), ((5, 3, 7), {}), ((4, 4, 7), {}), ((2, 2, 106), {}),
         ((4, 7, 7), FORCED(320)), ((4, 7, 7), FORCED(160)), ((3, 3, 9), FORCED(16)), ((2, 3, 5), FORCED(7))]


def problem(n, seed):
    from idp_gb300 import meshgen

    X0, tets = meshgen.bar(*n, size=tuple(0.25 * k for k in n), jitter=0.05, seed=seed)
    rng = np.random.default_rng(seed)
    return X0, tets, cases.problem(X0, tets), X0 + rng.uniform(-0.01, 0.01, X0.shape), rng.normal(size=X0.shape)


@pytest.mark.parametrize("mode", [0, 1], ids=["fp64", "mixed"])
@pytest.mark.parametrize("n,kw", SIZES, ids=lambda v: "x".join(map(str, v)) if isinstance(v, tuple) else "-".join(map(str, v.values())))
def test_direction_matches_direct_solve(oracle, gpu_lib, n, kw, mode):
    import idp_gb300 as idp
    import scipy.sparse.linalg as spla

    X0, tets, pr, X, v = problem(n, 1)
    V = X0.shape[0]
    dbc = np.array([0, V // 2], dtype=np.int32)
    X[dbc] = X0[dbc]
    ctx = ctx_for(idp, X0, tets, pr, mode, v=v, dbc=dbc, pcg_rel_tol=1e-8, **kw)
    p, its, rel = ctx.newton_direction(0, X)
    assert rel <= 1e-7 and its > 0
    pb = oracle_problem(oracle, X, tets, pr, X0=X0)
    cons, info = oracle.constraint_set(X, X0, oracle.surface(X0, tets), np.zeros(V, np.uint8), pr["dHat2"])
    assert len(cons) == 0
    H = oracle._hessian(pb, X, cons, info).tolil()
    g = oracle._gradient(pb, X, X0 + 0.1 * v, cons, info).reshape(-1)
    fixed = (3 * dbc[:, None] + np.arange(3)).reshape(-1)
    H[fixed, :] = 0
    H[:, fixed] = 0
    H[fixed, fixed] = 1
    g[fixed] = 0
    po = spla.spsolve(H.tocsc(), -g)
    assert np.linalg.norm(p - po) <= (1e-6 if mode == 0 else 2e-3) * np.linalg.norm(po)
    assert np.all(p.reshape(-1, 3)[dbc] == 0)
    ctx.close()


@pytest.mark.parametrize("mode", [0, 1], ids=["fp64", "mixed"])
def test_arena_bitwise_identical_to_alone(gpu_lib, mode):
    import idp_gb300 as idp

    probs = [problem(n, k) for k, n in enumerate([(5, 3, 7), (2, 2, 106), (1, 1, 2), (4, 4, 12)])]
    both = idp.Context(h=0.1, mode=mode)
    for X0, tets, pr, X, v in probs:
        both.add_instance(X0, tets, pr["mass"], pr["lam"], pr["mu"], pr["dHat2"], pr["kappa"], pr["kappa_max"])
    for i, q in enumerate(probs):
        both.set_velocity(i, 0.2 * q[4])
    both.commit()
    both.advance()
    for i, (X0, tets, pr, X, v) in enumerate(probs):
        alone = ctx_for(idp, X0, tets, pr, mode, v=0.2 * v)
        alone.advance()
        assert np.array_equal(alone.state(0)[0], both.state(i)[0]), i
        alone.close()
    both.close()
