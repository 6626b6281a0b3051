"""Kernels that work in tiles, at the edges of the tiles: energy sums and
gradients (64 to 256 elements per CTA, the last CTA of an instance finishes its
sum), FP64 Hessian products, the exact parallel sums behind the CCD's span cap,
and the sorts of constraint records, gradient and Hessian entries (tiles of
1,024 items up to 49,152, radix passes above).

Energies, gradients and FP64 Hessian products within 1e-9 relative of the
oracle, as the other parity tests; step bounds and constraint sets equal.
"""
import ctypes as C

import numpy as np
import pytest

import cases
from test_gpu_parity import ctx_for, oracle_problem, sort_rows
from test_zz_no_alloc import _dev, _rest

pytestmark = pytest.mark.gpu


def first_tets(T, seed):
    """T tets of a jittered bar and the vertices they use."""
    from idp_gb300 import meshgen

    X, tets = meshgen.bar(4, 4, 9, size=(1.0, 1.0, 2.25), jitter=0.05, seed=seed)
    used, local = np.unique(tets[:T], return_inverse=True)
    return X[used], local.reshape(-1, 4).astype(np.int32)


@pytest.mark.parametrize("T", [1, 63, 64, 65, 127, 128, 255, 256, 257, 513])
def test_energy_gradient_hessian(oracle, gpu_lib, T):
    import torch

    import idp_gb300 as idp

    X0, tets = first_tets(T, T)
    pr = cases.problem(X0, tets)
    rng = np.random.default_rng(T)
    X, v = X0 + rng.uniform(-0.01, 0.01, X0.shape), rng.normal(size=X0.shape)
    ctx = ctx_for(idp, X0, tets, pr, idp.MODE_FP64, v=v)
    pb = oracle_problem(oracle, X, tets, pr, X0=X0)
    xt = X0 + 0.1 * v
    cons, info = oracle.constraint_set(X, X0, oracle.surface(X0, tets), np.zeros(len(X0), np.uint8), pr["dHat2"])
    assert len(cons) == 0
    E_el = oracle.tet_energy(X, tets, pb.IB, pb.vol, pb.lam, pb.mu, 0.01)
    for _ in range(2):  # the second call must not see the first one's counters
        Ee, Ei, Eb = ctx.energy(0, X)
        assert Eb == 0 and Ee == pytest.approx(E_el, rel=1e-9)
        assert Ei == pytest.approx(0.5 * float(np.sum(pr["mass"][:, None] * (X - xt) ** 2)), rel=1e-9)
    go = oracle._gradient(pb, X, xt, cons, info)
    assert np.linalg.norm(ctx.gradient(0, X) - go) <= 1e-9 * np.linalg.norm(go)
    x = rng.normal(size=X.size)
    yo = oracle._hessian(pb, X, cons, info) @ x
    assert np.linalg.norm(ctx.hessian_apply(0, X, x) - yo) <= 1e-9 * np.linalg.norm(yo)
    ctx.close()
    IB, vol = _rest(X0, tets)
    a = [_dev(torch, tets, np.int32)] + [_dev(torch, k, np.float64) for k in
                                         (X, IB, vol, np.full(T, pr["lam"]), np.full(T, pr["mu"]))]
    e, bad = torch.zeros(1, dtype=torch.float64, device="cuda"), torch.zeros(1, dtype=torch.int32, device="cuda")
    for _ in range(2):
        assert gpu_lib.idp_tet_energy_noalloc(T, *[k.data_ptr() for k in a], 0.01, e.data_ptr(), bad.data_ptr(),
                                              C.c_void_p(torch.cuda.current_stream().cuda_stream)) == idp.IDP_OK
        assert int(bad.item()) == 0 and float(e.item()) == pytest.approx(E_el, rel=1e-9)


@pytest.mark.parametrize("n", [(1, 1, 1), (1, 1, 2), (3, 2, 5), (6, 6, 9), (9, 9, 40), (20, 20, 60)],
                         ids=lambda n: "x".join(map(str, n)))
@pytest.mark.parametrize("grid", [0.0, 0.05], ids=["equal_edges", "jittered"])
def test_span_cap(oracle, gpu_lib, n, grid):
    """A step through free space many voxels long: the span cap alone, from the
    Eigen-order sum of the edges and the serial sum of the displacements."""
    import idp_gb300 as idp
    from idp_gb300 import meshgen

    X, tets = meshgen.bar(*n, size=tuple(0.3 * k for k in n), jitter=grid, seed=2)
    ctx = ctx_for(idp, X, tets, cases.problem(X, tets), idp.MODE_MIXED)
    rng = np.random.default_rng(4)
    surf, z = oracle.surface(X, tets), np.zeros(X.shape[0], np.uint8)
    for d in (np.full(X.shape, 0.625), 0.7 + 1e-3 * rng.uniform(size=X.shape), np.tile([30.0, 0.0, 1 / 3], (len(X), 1))):
        ag, _ = ctx.ccd_stepsize(0, X, d.reshape(-1), 1.0)
        ao, rc = oracle.ccd_stepsize(X, d.reshape(-1), surf, z, 1.0)
        assert rc == 0 and ag == ao, (ag, ao)
    assert ag < 0.1
    ctx.close()


@pytest.mark.parametrize("n,dhat", [((1, 1, 2), 5e-3), ((2, 4, 8), 0.05), ((2, 9, 16), 0.08), ((1, 14, 24), 0.1)],
                         ids=["one_tile", "tiles", "more_tiles", "radix"])
def test_sorted_records_and_entries(oracle, gpu_lib, n, dhat):
    import idp_gb300 as idp

    X, tets = cases.two_bars(gap=2e-3, seed=3, n=n, shift=0.01)
    pr = cases.problem(X, tets, dHat=dhat)
    ctx = ctx_for(idp, X, tets, pr, idp.MODE_FP64)
    cons, info = oracle.constraint_set(X, X, oracle.surface(X, tets), np.zeros(len(X), np.uint8), pr["dHat2"])
    assert len(cons) > 0
    assert sort_rows(ctx.constraint_set(0, X)) == sort_rows(cons)
    pb = oracle_problem(oracle, X, tets, pr)
    go = oracle._gradient(pb, X, X, cons, info)
    assert np.linalg.norm(ctx.gradient(0, X) - go) <= 1e-9 * np.linalg.norm(go)
    x = np.random.default_rng(0).normal(size=X.size)
    yo = oracle._hessian(pb, X, cons, info) @ x
    assert np.linalg.norm(ctx.hessian_apply(0, X, x) - yo) <= 1e-9 * np.linalg.norm(yo)
    ctx.close()
