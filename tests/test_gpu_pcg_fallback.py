"""A contact-free body that does not fit the layout of the persistent PCG: a ball
whose tets all share the centre vertex, so that the CTA with the centre's row has
more halo vertices (4,098 surface vertices less its own rows) than its list holds.
It is solved by a thread-block cluster instead, and a bar beside it in the arena
still by the persistent CTAs.

Tolerances are those of the other direction tests: 1e-6 in FP64 (PCG to 1e-8
times the system's condition), 2e-3 in mixed mode (FP32 element Hessians).
"""
import numpy as np
import pytest

import cases
from test_gpu_parity import oracle_problem

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", [0, 1], ids=["fp64", "mixed"])
def test_body_with_a_hub(oracle, gpu_lib, mode):
    import idp_gb300 as idp
    import scipy.sparse.linalg as spla
    from idp_gb300 import meshgen

    S, F = cases.sphere_shell(levels=5)
    ball = np.concatenate([np.zeros((1, 3)), S]), np.concatenate([np.zeros((len(F), 1), int), F[:, [0, 2, 1]] + 1], 1)
    bar = meshgen.bar(3, 3, 9, size=(0.75, 0.75, 2.25), jitter=0.05, seed=1)
    rng = np.random.default_rng(2)
    ctx = idp.Context(h=0.1, mode=mode, pcg_rel_tol=1e-8)
    todo = []
    for X0, tets in (ball, bar):
        tets = np.ascontiguousarray(tets, dtype=np.int32)
        D = X0[tets[:, 1:]] - X0[tets[:, :1]]
        if np.linalg.det(D[0]) < 0:
            tets = np.ascontiguousarray(tets[:, [0, 1, 3, 2]])
        D = X0[tets[:, 1:]] - X0[tets[:, :1]]
        assert np.all(np.linalg.det(D) > 0)
        pr = cases.problem(X0, tets)
        v = rng.normal(size=X0.shape)
        i = ctx.add_instance(X0, tets, pr["mass"], pr["lam"], pr["mu"], pr["dHat2"], pr["kappa"], pr["kappa_max"])
        ctx.set_velocity(i, v)
        todo.append((i, X0, tets, pr, v, X0 + rng.uniform(-1e-3, 1e-3, X0.shape)))
    ctx.commit()
    for i, X0, tets, pr, v, X in todo:
        p, its, rel = ctx.newton_direction(i, X)
        assert rel <= 1e-7 and its > 0
        pb = oracle_problem(oracle, X, tets, pr, X0=X0)
        cons, info = oracle.constraint_set(X, X0, oracle.surface(X0, tets), np.zeros(len(X0), np.uint8), pr["dHat2"])
        assert len(cons) == 0
        H = oracle._hessian(pb, X, cons, info).tocsc()
        po = spla.spsolve(H, -oracle._gradient(pb, X, X0 + 0.1 * v, cons, info).reshape(-1))
        assert np.linalg.norm(p - po) <= (1e-6 if mode == 0 else 2e-3) * np.linalg.norm(po)
    ctx.close()
