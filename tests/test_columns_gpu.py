"""The column solves (vertical diffusion, the implicit part of a split w) at the sizes where
their block changes: 16 or 8 columns, shared memory above 48 KB, one lane per column or several
sharing one, tops below the surface, and members of different depth in one launch."""

import numpy as np
import pytest

from fesom_jax_b200 import inputs as I
from fesom_jax_b200 import meshgen
from tests.golden_cases import RTOL, cavity_mesh

DT = 1200.0


@pytest.fixture(scope="module")
def torch():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    return torch


@pytest.fixture(scope="module")
def meshes(pi):
    # 130 nodes: the last block is not full; bottoms from 3 levels on
    m = {nl: meshgen.make_mesh(130, nl=nl, bottom=(3, nl), seed=3) for nl in (12, 48, 70, 128)}
    return {**m, "cavity": cavity_mesh(pi)}


def _dev(torch, x):
    return torch.from_numpy(np.ascontiguousarray(x)).cuda()


def _Kv(m, rng):
    return rng.uniform(1e-5, 1e-2, (m.nod2D, m.nl)) * m.node_iface_mask


@pytest.mark.gpu
# shared memory of a block: 48 x 5 needs 50 KB, 48 x 8 and 70 x 8 take 8 columns (34 and 50 KB),
# 128 x 8 the most there is (91 KB); 2, 3, 7: lanes of a column with unequal shares
@pytest.mark.parametrize("nl,ntr", [(12, 8), (48, 2), (48, 3), (48, 5), (48, 8), (70, 7),
                                    (70, 8), (128, 1), (128, 8), (48, 11), ("cavity", 5)])
@pytest.mark.parametrize("scale", [1.0, 1e-300])   # 1e-300: rows the fast quotient refuses
def test_vertical_diffusion(torch, meshes, nl, ntr, scale):
    from fesom_jax_b200.tracer_diff import impl_vert_diff_one
    from oracle import vdiff_np
    m = meshes[nl]
    rng = np.random.default_rng(ntr)
    hnode, _ = I.rest_thickness(m)
    T = scale * rng.uniform(0.0, 20.0, (ntr, m.nod2D, m.nl))
    Kv, bc = _Kv(m, rng), scale * rng.normal(0.0, 0.01, (ntr, m.nod2D))
    up = [_dev(torch, x) for x in (T, Kv, hnode, bc)]
    got = impl_vert_diff_one(m, up[0], up[1], up[2], dt=DT, bc_surf=up[3])
    inplace = up[0].clone()
    from fesom_jax_b200.tracer_diff import _run
    _run(m, inplace, up[1], up[2], DT, up[3], None, None, out=inplace)
    assert torch.equal(inplace, got)
    for t in range(ntr):
        one = impl_vert_diff_one(m, up[0][t], up[1], up[2], dt=DT, bc_surf=up[3][t])
        assert torch.equal(got[t], one)      # several tracers: the bits of separate solves
        ref = vdiff_np.impl_vert_diff_one(m, T[t], Kv, hnode, dt=DT, bc_surf=bc[t])
        x = one.cpu().numpy()
        assert np.max(np.abs(x - ref)) <= RTOL * np.max(np.abs(ref))
        assert np.array_equal(x[~m.node_layer_mask], T[t][~m.node_layer_mask])


@pytest.mark.gpu
@pytest.mark.parametrize("nl,ntr", [(12, 3), (48, 5), (70, 8), ("cavity", 3), ("cavity", 5)])
def test_split_w_and_moving_depths(torch, meshes, nl, ntr):
    """A step with w_i, Z3d and zbar3 on the small-mesh path and its stage-by-stage form."""
    from fesom_jax_b200.tracer_adv import FctPlan
    from oracle import fct_np
    m = meshes[nl]
    f = I.make_fields(m, seed=ntr, n_passive=6, ab2=True, kind="psi" if nl == "cavity" else "basin")
    zbar3 = np.broadcast_to(m.zbar, (m.nod2D, m.nl)).copy()
    zbar3[:, 1:] *= 1.0 + 0.01 * np.sin(np.arange(m.nod2D))[:, None]
    Z3d = np.concatenate([0.5 * (zbar3[:, :-1] + zbar3[:, 1:]),
                          0.5 * (zbar3[:, -2:-1] + zbar3[:, -1:])], axis=1)
    w_i = 0.3 * f.w_e
    T, To = f.tracers[:ntr], f.tracers_old[:ntr]
    args = [_dev(torch, x) for x in (f.uv, f.w_e - w_i, f.helem, f.hnode, f.hnode_new, T, To)]
    kw = dict(zip(("Z3d", "zbar3", "w_i"), (_dev(torch, x) for x in (Z3d, zbar3, w_i))))
    plan = FctPlan(m, 0, max_tracers=ntr)
    plan.fill_workspace(0xFF)
    got = plan.forward(*args, DT, **kw).cpu().numpy()
    plan.set_mapping(1, 2)               # the run kernels: the same bits
    assert np.array_equal(plan.forward(*args, DT, **kw).cpu().numpy(), got)
    plan.set_fused(False)
    stages = plan.forward(*args, DT, **kw).cpu().numpy()
    plan.close()
    lm = m.node_layer_mask
    for t in range(ntr):
        ref, _ = fct_np.advect_one_fct(m, f.uv, f.w_e - w_i, f.helem, f.hnode, f.hnode_new, T[t],
                                       To[t], dt=DT, Z3d=Z3d, zbar3=zbar3, w_i=w_i)
        for x in (got[t], stages[t]):
            assert np.max(np.abs(x - ref)[lm]) <= RTOL * np.max(np.abs(ref[lm]))


@pytest.mark.gpu
@pytest.mark.parametrize("ntr", [5, 8])
def test_batched_epilogue_of_members_of_different_depth(torch, meshes, ntr):
    """Kv members of 128, 12, 48 and 70 levels in one launch: the bits of plain steps, each
    followed by the diffusion call."""
    from fesom_jax_b200.ensemble import Ensemble
    from fesom_jax_b200.tracer_adv import get_plan
    from fesom_jax_b200.tracer_diff import impl_vert_diff_one
    ens, want = Ensemble(), []
    for i, nl in enumerate((128, 12, 48, 70)):
        m = meshes[nl]
        f = I.make_fields(m, seed=i, n_passive=6, ab2=True, kind="basin")
        a = [_dev(torch, x) for x in (f.uv, f.w_e, f.helem, f.hnode, f.hnode_new)]
        T, To = (_dev(torch, x[:ntr]) for x in (f.tracers, f.tracers_old))
        Kv = _dev(torch, _Kv(m, np.random.default_rng(i)))
        ens.add_member(m, *a, T, To, DT, Kv=Kv)
        for _ in range(2):
            T, To = impl_vert_diff_one(m, get_plan(m, 0).forward(*a, T, To, DT), Kv, a[4],
                                       dt=DT), T
        want.append((T, To))
    ens.build()
    ens.run(2)
    for i, (T, To) in enumerate(want):
        got, old = ens.state(i)
        assert torch.equal(got, T) and torch.equal(old, To)
    ens.close()


@pytest.mark.gpu
@pytest.mark.parametrize("ntr", [8, 10, 16])
def test_batched_epilogue_of_many_columns(torch, meshes, ntr):
    """Enough columns for the walks of eight tracers (chunks of 8, 8 + 2 and 8 + 8), members of
    12 to 128 levels and a cavity in one launch: the bits of plain steps and diffusion calls."""
    from fesom_jax_b200.ensemble import Ensemble
    from fesom_jax_b200.tracer_adv import get_plan
    from fesom_jax_b200.tracer_diff import impl_vert_diff_one
    ens, want = Ensemble(), []
    order = ("cavity", 128, 12, "cavity", 48, 70, "cavity", 12)
    assert len(order) * meshes["cavity"].nod2D >= 148 * 5 * 256 // 8
    for i, nl in enumerate(order):
        m = meshes[nl]
        f = I.make_fields(m, seed=i, n_passive=ntr - 2, ab2=True,
                          kind="psi" if nl == "cavity" else "basin")
        a = [_dev(torch, x) for x in (f.uv, f.w_e, f.helem, f.hnode, f.hnode_new)]
        T, To = (_dev(torch, x) for x in (f.tracers, f.tracers_old))
        Kv = _dev(torch, _Kv(m, np.random.default_rng(i)))
        ens.add_member(m, *a, T, To, DT, Kv=Kv)
        for _ in range(2):
            T, To = impl_vert_diff_one(m, get_plan(m, 0).forward(*a, T, To, DT), Kv, a[4],
                                       dt=DT), T
        want.append((T, To))
    ens.build()
    ens.fill_workspace(0xFF)
    ens.run(2)
    assert ens.info()["groups"] == 1
    for i, (T, To) in enumerate(want):
        got, old = ens.state(i)
        assert torch.equal(got, T) and torch.equal(old, To)
    ens.close()
