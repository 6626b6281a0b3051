"""The broad phases' far tests and their fused queries: constraint sets and CCD
step bounds must be the oracle's bit for bit where the FP32 filter has least
room: large coordinates, small and stretched scenes (sliver triangles, nearly
parallel edges), gaps at the activation distance, zero, grazing and head-on
directions, first and later builds, alone and beside other instances. No
tolerance: sets and step bounds are compared for equality.
"""
import numpy as np
import pytest

import cases
from test_gpu_parity import ctx_for, sort_rows

pytestmark = pytest.mark.gpu

FORMS = {
    "plain": (1.0, 0.0),
    "shifted": (1.0, np.array([1e3, -2e3, 500.0])),
    "small": (1e-3, 0.0),
    "large": (1e3, np.array([0.0, 1e5, 0.0])),
    "flat": (np.array([1.0, 1e-3, 1.0]), 0.0),
    "long": (np.array([1.0, 1.0, 300.0]), 7.0),
}


def scene(form, seed):
    X, tets = cases.two_bars(gap=2e-3, seed=seed)
    scale, shift = FORMS[form]
    gap = 2e-3 * (scale if np.ndim(scale) == 0 else scale[0])
    return X * scale + shift, tets, gap


@pytest.mark.parametrize("form", sorted(FORMS))
def test_constraint_set_at_the_activation_distance(oracle, gpu_lib, form):
    import idp_gb300 as idp

    X, tets, gap = scene(form, 1)
    surf = oracle.surface(X, tets)
    z = np.zeros(X.shape[0], np.uint8)
    half = X.shape[0] // 2
    for d in (gap * (1 - 1e-9), gap * (1 + 1e-9), 1.7 * gap):
        pr = cases.problem(X, tets, dHat=d)
        ctx = ctx_for(idp, X, tets, pr, idp.MODE_MIXED)
        for push in (0.0, 0.3, 0.0):  # of the gap
            Y = X.copy()
            Y[half:, 0] -= push * gap
            o, _ = oracle.constraint_set(Y, X, surf, z, pr["dHat2"])
            assert sort_rows(ctx.constraint_set(0, Y)) == sort_rows(o), (d / gap, push)
        ctx.close()
    assert len(o) > 0


@pytest.mark.parametrize("form", sorted(FORMS))
def test_ccd_of_zero_grazing_and_head_on_steps(oracle, gpu_lib, form):
    import idp_gb300 as idp

    X, tets, gap = scene(form, 2)
    surf = oracle.surface(X, tets)
    z = np.zeros(X.shape[0], np.uint8)
    half = X.shape[0] // 2
    rng = np.random.default_rng(3)
    ctx = ctx_for(idp, X, tets, cases.problem(X, tets, dHat=gap), idp.MODE_MIXED)
    for k, (vx, vy, noise) in enumerate([(0, 0, 0), (0, 2, 0), (-0.9, 1, 0), (-1.2, 0, 0), (-40, 0, 0), (-3, 1, 2), (30, 0, 0)]):
        d = noise * gap * rng.normal(size=X.shape)
        d[half:, 0] += vx * gap
        d[half:, 1] += vy * gap
        for a0 in (1.0, 0.37):
            ag, _ = ctx.ccd_stepsize(0, X, d.reshape(-1), a0)
            ao, rc = oracle.ccd_stepsize(X, d.reshape(-1), surf, z, a0)
            assert rc == 0 and ag == ao, (k, a0, ag, ao)
    ctx.close()


def test_instances_of_unlike_scales_side_by_side(oracle, gpu_lib):
    import idp_gb300 as idp

    ctx = idp.Context(h=0.1, mode=idp.MODE_MIXED)
    parts = []
    for i, form in enumerate(sorted(FORMS)):
        X, tets, gap = scene(form, i)
        pr = cases.problem(X, tets, dHat=1.5 * gap)
        ctx.add_instance(X, tets, pr["mass"], pr["lam"], pr["mu"], pr["dHat2"], pr["kappa"], pr["kappa_max"])
        parts.append((X, tets, gap, pr))
    ctx.commit()
    for i, (X, tets, gap, pr) in enumerate(parts):
        surf = oracle.surface(X, tets)
        z = np.zeros(X.shape[0], np.uint8)
        o, _ = oracle.constraint_set(X, X, surf, z, pr["dHat2"])
        assert len(o) > 0 and sort_rows(ctx.constraint_set(i, X)) == sort_rows(o)
        d = np.zeros_like(X)
        d[X.shape[0] // 2:, 0] = -3 * gap
        ag, _ = ctx.ccd_stepsize(i, X, d.reshape(-1), 1.0)
        assert ag == oracle.ccd_stepsize(X, d.reshape(-1), surf, z, 1.0)[0] and ag < 1
    ctx.close()
