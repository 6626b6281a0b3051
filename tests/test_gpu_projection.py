"""PSD projection of the barrier's and the shells' element Hessians (16 lanes
per matrix, sizes 6, 9 and 12 mixed in one launch): Hessian products against
the oracle's, over contact configurations that hold point-point, point-edge,
point-triangle and edge-edge stencils.

Tolerances: FP64 1e-9 of the product. Mixed mode: a stored block is off by its
rounding (6e-8), the projection (below 12 eps of the matrix norm) and the
assembly's sums (about 10 eps): under 2e-6 of |H| |x|; 1e-5 is asked.
"""
import numpy as np
import pytest

import cases
from test_gpu_parity import contact_configs, ctx_for, oracle_problem

pytestmark = pytest.mark.gpu


def stencil_sizes(cons):
    """6, 9 or 12 per record (sign encoding of FEM/IPC.h:202-250)."""
    return {12 if c[0] >= 0 or c[3] >= 0 else (9 if c[2] >= 0 else 6) for c in np.asarray(cons)}


def configs():
    X, tets = cases.two_bars(gap=2e-2, seed=0)
    return contact_configs() + [("two_bars_wide", X, tets, X, 0.2)]


@pytest.mark.parametrize("mode", [0, 1], ids=["fp64", "mixed"])
@pytest.mark.parametrize("k,sizes", [(0, {12}), (4, {6, 9, 12}), (5, {9, 12})], ids=["n12", "n6_9_12", "n9_12"])
def test_projected_hessian_product(oracle, gpu_lib, k, sizes, mode):
    import idp_gb300 as idp

    name, X0, tets, X, dhat = configs()[k]
    pr = cases.problem(X0, tets, dHat=dhat)
    ctx = ctx_for(idp, X0, tets, pr, mode)
    pb = oracle_problem(oracle, X, tets, pr, X0=X0)
    cons, info = oracle.constraint_set(X, X0, oracle.surface(X0, tets), np.zeros(X0.shape[0], np.uint8), pr["dHat2"])
    assert stencil_sizes(cons) == sizes
    H = oracle._hessian(pb, X, cons, info)
    rng = np.random.default_rng(k)
    for _ in range(2):
        x = rng.normal(size=X.size)
        y, yo = ctx.hessian_apply(0, X, x), H @ x
        bound = 1e-9 * np.linalg.norm(yo) if mode == 0 else 1e-5 * np.linalg.norm(abs(H) @ np.abs(x))
        assert np.linalg.norm(y - yo) <= bound
    ctx.close()


def test_projection_does_not_depend_on_its_neighbours(oracle, gpu_lib):
    """A context's Hessian product is bit for bit the same beside other
    instances (matrices share warps with other instances' matrices there)."""
    import idp_gb300 as idp

    probs = []
    for k in (0, 4, 5):
        name, X0, tets, X, dhat = configs()[k]
        probs.append((X0, tets, X, cases.problem(X0, tets, dHat=dhat)))
    both = idp.Context(h=0.1, mode=idp.MODE_MIXED)
    for X0, tets, X, pr in probs:
        both.add_instance(X0, tets, pr["mass"], pr["lam"], pr["mu"], pr["dHat2"], pr["kappa"], pr["kappa_max"])
    both.commit()
    rng = np.random.default_rng(3)
    for i, (X0, tets, X, pr) in enumerate(probs):
        x = rng.normal(size=X.size)
        alone = ctx_for(idp, X0, tets, pr, idp.MODE_MIXED)
        assert np.array_equal(alone.hessian_apply(0, X, x), both.hessian_apply(i, X, x))
        alone.close()
    both.close()
