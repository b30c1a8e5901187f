"""What a step derives from uv: w on meshes whose edges reach beyond their end nodes' layers,
and the volume fluxes and w of a multi-step run, formed from the uv it finds at its start."""

import numpy as np
import pytest

from fesom_jax_b200 import inputs as I
from fesom_jax_b200 import meshgen
from fesom_jax_b200.mesh import FCT_FIELDS, Mesh
from tests.golden_cases import RTOL, cavity_mesh

DT = 1200.0


@pytest.fixture(scope="module")
def torch():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    return torch


def _dev(torch, x):
    return torch.from_numpy(np.ascontiguousarray(x)).cuda()


def _edges_outside(m):
    """``m`` with every seventh node two levels shallower, and every eleventh starting one
    level lower, than its cells."""
    fields = {f: np.array(getattr(m, f)) for f in FCT_FIELDS}
    n = fields["nlevels_nod2D"]
    n[::7] = np.maximum(n[::7] - 2, fields["ulevels_nod2D"][::7])
    u = fields["ulevels_nod2D"]
    u[::11] = np.minimum(u[::11] + 1, n[::11])
    return Mesh(**fields, name=m.name + "_edges_outside")


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["plain", "cavity", "edges_outside"])
def test_compute_w(torch, pi, kind):
    from fesom_jax_b200.ale import compute_w
    m = cavity_mesh(pi) if kind == "cavity" else meshgen.make_mesh(700, nl=33, bottom=(3, 33),
                                                                  seed=3)
    rng = np.random.default_rng(0)
    uv = rng.normal(0.0, 0.1, (m.elem2D, m.nl, 2))
    _, helem = I.rest_thickness(m)
    if kind == "edges_outside":
        m = _edges_outside(m)
        lm, em = m.node_layer_mask, m.elem_layer_mask
        outside = em[m.edge_tri[:, 0]][:, None] & ~lm[m.edges]
        assert outside.any(axis=(1, 2)).sum() > 100
    ref = I.compute_w(m, uv, helem)
    got = compute_w(m, _dev(torch, uv), _dev(torch, helem)).cpu().numpy()
    assert np.max(np.abs(got - ref)) <= RTOL * np.max(np.abs(ref))
    assert np.all(got[~m.node_iface_mask] == 0.0)


@pytest.mark.gpu
@pytest.mark.parametrize("derive_w", [False, True])
def test_each_run_takes_the_uv_it_starts_from(torch, derive_w):
    """A new uv written into a member's array between two launches of the same cached graph,
    and before a single step: the bits of plain steps with that uv."""
    from fesom_jax_b200.ale import compute_w
    from fesom_jax_b200.ensemble import Ensemble
    from fesom_jax_b200.tracer_adv import get_plan
    m = meshgen.make_mesh(700, nl=33, bottom=(3, 33), seed=3)
    fs = [I.make_fields(m, seed=s, ab2=True, kind="basin") for s in (1, 2, 3)]
    f = fs[0]
    w, helem, hnode, hnode_new = (_dev(torch, x) for x in (f.w_e, f.helem, f.hnode, f.hnode_new))
    T, To = _dev(torch, f.tracers), _dev(torch, f.tracers_old)
    ens = Ensemble()
    ens.add_member(m, _dev(torch, f.uv), None if derive_w else w, helem, hnode, hnode_new, T, To,
                   DT, derive_w=derive_w)
    ens.build()
    for g, steps in zip(fs, (3, 3, 1)):
        uv = _dev(torch, g.uv)
        ens.members[0].uv.copy_(uv)
        if steps > 1:
            ens.run(steps)
        else:
            ens.step()
        we = compute_w(m, uv, helem) if derive_w else w
        for _ in range(steps):
            T, To = get_plan(m, 0).forward(uv, we, helem, hnode, hnode_new, T, To, DT), T
        got, old = ens.state(0)
        assert torch.equal(got, T) and torch.equal(old, To)
    ens.close()
