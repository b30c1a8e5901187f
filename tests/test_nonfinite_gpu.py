"""Where a NaN of the input reaches: T_new is non-finite where the scheme's stencil takes the
value, and stays finite elsewhere."""

import numpy as np
import pytest

from fesom_jax_b200 import inputs as I
from fesom_jax_b200 import meshgen

DT = 1200.0


@pytest.fixture(scope="module")
def torch():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    return torch


@pytest.fixture(scope="module")
def case():
    """A mesh, fields, and a dozen wet (node, level) places far from one another."""
    m = meshgen.make_mesh(4000, nl=20, bottom=(4, 20), seed=2)
    f = I.make_fields(m, seed=2, n_passive=1, ab2=True, kind="basin")
    rng = np.random.default_rng(1)
    free, places = np.ones(m.nod2D, bool), []
    while len(places) < 12:
        v = int(rng.choice(np.flatnonzero(free)))
        places.append((v, int(rng.integers(0, m.nlevels_nod2D[v] - 1))))
        free &= _distance(m, v, 9) > 8
    return m, f, places


def _distance(m, v, most):
    d = np.full(m.nod2D, most)
    d[v] = 0
    for r in range(1, most):
        for a, b in ((0, 1), (1, 0)):
            near = m.edges[d[m.edges[:, a]] == r - 1, b]
            d[near] = np.minimum(d[near], r)
    return d


def _dev(torch, x):
    return torch.from_numpy(np.ascontiguousarray(x)).cuda()


def _with_nan(f, places):
    T = f.tracers.copy()
    for v, k in places:
        T[:, v, k] = np.nan
    return T


@pytest.mark.gpu
@pytest.mark.parametrize("mapping", [None, (1, 1), (2, 2), (2, 4), "batch"])
def test_fused_step_keeps_a_nan_within_its_stencil(torch, case, mapping):
    """LO of v's neighbours is NaN at its level, their fluxes carry it one node further there.
    The bounds pass over it, so two nodes away the levels above and below stay finite."""
    from fesom_jax_b200.ensemble import Ensemble
    from fesom_jax_b200.tracer_adv import FctPlan
    m, f, places = case
    args = [_dev(torch, x) for x in (f.uv, f.w_e, f.helem, f.hnode, f.hnode_new)]
    T, To = _dev(torch, _with_nan(f, places)), _dev(torch, f.tracers_old)
    if mapping == "batch":
        ens = Ensemble()
        ens.add_member(m, *args, T, To, DT)
        ens.build()
        ens.run(1)
        got = ens.state(0)[0].cpu().numpy()
        ens.close()
    else:
        plan = FctPlan(m, 0, max_tracers=3)
        if mapping:
            plan.set_mapping(*mapping)
        got = plan.forward(*args, T, To, DT).cpu().numpy()
        plan.close()
    allowed = np.zeros((m.nod2D, m.nl), bool)
    for v, k in places:
        d = _distance(m, v, 4)
        allowed[d <= 1] = True
        allowed[d == 2, k] = True
        assert not np.isfinite(got[:, v, k]).any()
    bad = ~np.isfinite(got)
    assert not (bad & ~allowed[None]).any()


def _reached(m, places):
    """Edge levels whose flux formula holds a NaN of ``places``: a vertex of the up or down cell
    (where MFCT takes the cells), or of a cell around either end node (elsewhere)."""
    from oracle import fct_np
    T = np.zeros((m.nod2D, m.nl))
    for v, k in places:
        T[v, k] = np.nan
    with np.errstate(invalid="ignore"):
        g = fct_np.fill_up_dn_grad(m, fct_np.tracer_gradient_elements(m, T))
    hit = ~np.isfinite(np.asarray(g)).all(axis=tuple(
        a for a in range(np.ndim(g)) if np.shape(g)[a] not in (m.edge2D, m.nl)))
    assert hit.shape == (m.edge2D, m.nl) and hit.sum() > 100
    k = np.arange(m.nl)[None, :]
    wet = np.zeros(hit.shape, bool)
    for j in range(2):
        el = m.edge_tri[:, j]
        wet |= (el >= 0)[:, None] & (k >= (m.ulevels[el] - 1)[:, None]) & \
            (k < (m.nlevels[el] - 1)[:, None])
    return hit & wet


@pytest.mark.gpu
@pytest.mark.parametrize("stagewise", [False, True])
def test_a_nan_of_either_gradient_reaches_both_ends(torch, case, stagewise):
    """The flux weighs the downwind end's gradient with 0, and 0 x NaN is NaN: T_new of both
    ends is non-finite, in the fused step (by way of LO and the limiter) and stage by stage."""
    from fesom_jax_b200.tracer_adv import FctPlan
    m, f, places = case
    plan = FctPlan(m, 0, max_tracers=3)
    plan.set_fused(not stagewise)
    got = plan.forward(*(_dev(torch, x) for x in (f.uv, f.w_e, f.helem, f.hnode, f.hnode_new,
                                                  _with_nan(f, places), f.tracers_old)),
                       DT).cpu().numpy()
    plan.close()
    e, k = np.nonzero(_reached(m, places))
    for end in range(2):
        assert not np.isfinite(got[:, m.edges[e, end], k]).any()


@pytest.mark.gpu
@pytest.mark.parametrize("tape", [False, True])
def test_a_nan_of_either_gradient_reaches_the_velocity_gradient(torch, case, tape):
    """The limiter's sums of both ends have a NaN cotangent then, which the uv of every cell
    around them receives."""
    from fesom_jax_b200.adjoint import Tape, advect_one_fct_vjp
    m, f, places = case
    args = [_dev(torch, x) for x in (f.uv, f.w_e, f.helem, f.hnode, f.hnode_new,
                                     _with_nan(f, places)[0], f.tracers_old[0])]
    kw = {}
    if tape:
        kw["tape"] = Tape(m, 1)
        kw["tape"].forward(0, *args, DT)
    guv = advect_one_fct_vjp(m, *args, torch.ones_like(args[5]), dt=DT, **kw)[2].cpu().numpy()
    e, k = np.nonzero(_reached(m, places))
    near = np.zeros((m.nod2D, m.nl), bool)
    for end in range(2):
        near[m.edges[e, end], k] = True
    kk = np.arange(m.nl)[None, :]
    wet = (kk >= (m.ulevels - 1)[:, None]) & (kk < (m.nlevels - 1)[:, None])
    cells = near[m.elem_nodes].any(axis=1) & wet
    assert cells.sum() > 100 and not np.isfinite(guv[cells]).any()
