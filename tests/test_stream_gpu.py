"""The stream kernels and their dispatch at the sizes where it changes: tracer counts that
split into pairs, fours, single slices and several launches; instances smaller and larger than
the resident grid; single instances on either side of the one-launch first stages; column
solves of one to nine tracers."""

import numpy as np
import pytest

from fesom_jax_b200 import inputs as I
from fesom_jax_b200 import meshgen

DT = 1200.0
RTOL = 1e-12   # the per-step tolerance of the C oracle tests


@pytest.fixture(scope="module")
def torch():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    return torch


@pytest.fixture(scope="module")
def meshes():
    return {n: meshgen.make_mesh(n, nl=nl, bottom=(3, nl), seed=3)
            for n, nl in ((90, 5), (700, 33), (9000, 48))}


def _dev(torch, x):
    return torch.from_numpy(np.ascontiguousarray(x)).cuda()


def _oracle(mesh, f, T, To):
    from oracle import fct_c
    return fct_c.advect_one_fct(mesh, f.uv, f.w_e, f.helem, f.hnode, f.hnode_new, T, To, dt=DT)[0]


@pytest.mark.gpu
@pytest.mark.parametrize("nodes", [90, 700, 9000])
@pytest.mark.parametrize("ntr", [1, 2, 3, 5])
def test_single_instance_matches_oracle(torch, meshes, nodes, ntr):
    from fesom_jax_b200.tracer_adv import FctPlan
    m = meshes[nodes]
    f = I.make_fields(m, seed=ntr, n_passive=max(0, ntr - 2), ab2=True, kind="basin")
    T, To = f.tracers[:ntr].copy(), f.tracers_old[:ntr].copy()
    T[:, ~m.node_layer_mask] = 7.5       # dry levels keep T
    plan = FctPlan(m, 0, max_tracers=ntr)
    args = [_dev(torch, x) for x in (f.uv, f.w_e, f.helem, f.hnode, f.hnode_new, T, To)]
    plan.fill_workspace(0xFF)            # NaN: nothing unwritten is read
    got = plan.forward(*args, DT).cpu().numpy()
    for t in range(ntr):
        ref = _oracle(m, f, T[t], To[t])
        assert np.max(np.abs(got[t] - ref)) <= RTOL * np.max(np.abs(ref))
        assert np.all(got[t][~m.node_layer_mask] == 7.5)
    plan.set_mapping(2, 2)               # the run kernels: the same bits
    assert np.array_equal(plan.forward(*args, DT).cpu().numpy(), got)
    plan.close()


@pytest.mark.gpu
@pytest.mark.parametrize("ntr", [1, 2, 3, 4, 5, 6, 7, 8, 10])
def test_members_equal_single_calls(torch, meshes, ntr):
    from fesom_jax_b200.ensemble import Ensemble
    from fesom_jax_b200.tracer_adv import get_plan
    ens, want = Ensemble(), []
    for i, n in enumerate((90, 9000, 700, 700)):
        m = meshes[n]
        f = I.make_fields(m, seed=10 * ntr + i, n_passive=max(0, ntr - 2), ab2=True,
                          kind="basin")
        T, To = f.tracers[:ntr], f.tracers_old[:ntr]
        ens.add_member(m, f.uv, f.w_e, f.helem, f.hnode, f.hnode_new, T, To, DT)
        args = [_dev(torch, x) for x in (f.uv, f.w_e, f.helem, f.hnode, f.hnode_new)]
        T, To = _dev(torch, T), _dev(torch, To)
        for _ in range(3):
            T, To = get_plan(m, 0).forward(*args, T, To, DT), T
        want.append((T.cpu().numpy(), To.cpu().numpy()))
    ens.build()
    ens.fill_workspace(0xFF)
    ens.run(3)
    for mapping in (None, (4, 1), (1, 1), (2, 4)):
        if mapping is not None:          # one more step under another mapping: the same bits
            ref = [ens.state(i)[0].clone() for i in range(4)]
            old = [ens.state(i)[1].clone() for i in range(4)]
            ens.step()
            a = [ens.state(i)[0].clone() for i in range(4)]
            for i in range(4):
                ens.set_state(i, ref[i], old[i])
            ens.set_mapping(*mapping)
            ens.step()
            for i in range(4):
                assert torch.equal(ens.state(i)[0], a[i])
            continue
        for i, (T, To) in enumerate(want):
            got, got_old = (x.cpu().numpy() for x in ens.state(i))
            assert np.array_equal(got, T) and np.array_equal(got_old, To)
    ens.close()


@pytest.mark.gpu
@pytest.mark.parametrize("ntr", [1, 2, 8, 9])
@pytest.mark.parametrize("nodes", [90, 700])
def test_column_solves_match_oracle(torch, meshes, nodes, ntr):
    from fesom_jax_b200.tracer_diff import impl_vert_diff_one
    from oracle import vdiff_np
    m = meshes[nodes]
    rng = np.random.default_rng(ntr)
    hnode, _ = I.rest_thickness(m)
    T = rng.uniform(0.0, 20.0, (ntr, m.nod2D, m.nl))
    Kv = rng.uniform(1e-5, 1e-2, (m.nod2D, m.nl)) * m.node_iface_mask
    bc = rng.normal(0.0, 0.01, (ntr, m.nod2D))
    got = impl_vert_diff_one(m, T, Kv, hnode, dt=DT, bc_surf=bc)
    for t in range(ntr):
        ref = vdiff_np.impl_vert_diff_one(m, T[t], Kv, hnode, dt=DT, bc_surf=bc[t])
        assert np.max(np.abs(got[t] - ref)) <= RTOL * np.max(np.abs(ref))
