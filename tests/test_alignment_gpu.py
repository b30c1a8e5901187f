"""Field pointers that start at an odd double of a larger buffer (8-byte aligned views)."""

import numpy as np
import pytest

from fesom_jax_b200 import inputs as I
from fesom_jax_b200 import meshgen


@pytest.fixture(scope="module")
def torch():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    return torch


@pytest.fixture(scope="module")
def mesh():
    return meshgen.make_mesh(700, nl=33, bottom=(3, 33), seed=3)


def _at(torch, x, offset):
    """``x`` on the GPU, ``offset`` doubles into its buffer (contiguous)."""
    x = torch.from_numpy(np.ascontiguousarray(x))
    buf = torch.empty(x.numel() + offset, dtype=torch.float64, device="cuda")
    v = buf[offset:].view(x.shape)
    v.copy_(x)
    assert v.is_contiguous() and v.data_ptr() % 16 == 8 * (offset % 2)
    return v


@pytest.mark.gpu
@pytest.mark.parametrize("offset", [1, 2, 3])
def test_compute_w_takes_uv_at_any_double(torch, mesh, offset):
    from fesom_jax_b200.ale import compute_w
    f = I.make_fields(mesh, seed=4, kind="basin")
    helem = _at(torch, f.helem, offset)
    want = compute_w(mesh, _at(torch, f.uv, 0), helem)
    got = compute_w(mesh, _at(torch, f.uv, offset), helem)
    assert torch.equal(got, want)


@pytest.mark.gpu
def test_step_refuses_uv_off_a_16_byte_boundary(torch, mesh):
    """The volume-flux kernel reads (u, v) pairs: every call that launches it refuses such a
    pointer on the host; the reverse pass of a taped step, which does not read uv, takes it."""
    from fesom_jax_b200.adjoint import Tape, advect_one_fct_vjp
    from fesom_jax_b200.ensemble import Ensemble
    from fesom_jax_b200.tracer_adv import FctPlan
    f = I.make_fields(mesh, seed=4, kind="basin")
    uv, off = _at(torch, f.uv, 0), _at(torch, f.uv, 1)
    rest = [_at(torch, x, 1) for x in (f.w_e, f.helem, f.hnode, f.hnode_new, f.tracers[0],
                                       f.tracers_old[0])]
    plan = FctPlan(mesh, 0)
    want = plan.forward(uv, *rest, 1200.0)      # the other fields may start anywhere
    for kw in ({}, {"stagewise": True}):
        if kw:
            plan.set_fused(False)
        with pytest.raises(Exception, match="16-byte"):
            plan.forward(off, *rest, 1200.0, **kw)
    plan.set_fused(True)
    assert torch.equal(plan.forward(uv, *rest, 1200.0), want)
    plan.close()
    ens = Ensemble()
    ens.add_member(mesh, off, *rest[:4], rest[4], rest[5], 1200.0)
    with pytest.raises(Exception, match="16-byte"):
        ens.build()
    g = torch.ones_like(rest[4])
    with pytest.raises(Exception, match="16-byte"):
        advect_one_fct_vjp(mesh, off, *rest, g, dt=1200.0)
    with Tape(mesh, 1) as tape:
        with pytest.raises(Exception, match="16-byte"):
            tape.forward(0, off, *rest, 1200.0)
        tape.forward(0, uv, *rest, 1200.0)
        a = advect_one_fct_vjp(mesh, uv, *rest, g, dt=1200.0, tape=tape)
        b = advect_one_fct_vjp(mesh, off, *rest, g, dt=1200.0, tape=tape)
        assert all(torch.equal(x, y) for x, y in zip(a, b))


@pytest.mark.gpu
@pytest.mark.parametrize("ntr", [2, 4])
def test_batch_takes_tracer_buffers_at_any_double(torch, mesh, ntr):
    """Interleaved buffers off a 16-byte boundary: single loads instead of tracer pairs, the
    same bits under the default mapping and a set one, batched and served."""
    import ctypes as C
    from fesom_jax_b200 import _lib
    from fesom_jax_b200.ensemble import FctInstance, _bind_batch
    from fesom_jax_b200.serve import _bind
    from fesom_jax_b200.tracer_adv import get_plan
    f = I.make_fields(mesh, seed=4, n_passive=2, ab2=True, kind="basin")
    fields = [_at(torch, x, 0) for x in (f.uv, f.w_e, f.helem, f.hnode, f.hnode_new)]
    old, T = (np.moveaxis(x[:ntr], 0, -1) for x in (f.tracers_old, f.tracers))
    L, plan = _bind_batch(_lib.lib()), get_plan(mesh, 0)
    s = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    got = []
    for offset in (0, 1):
        for run in ("batch", "mapped", "serve"):
            buf = [_at(torch, x, offset) for x in (old, T, T)]
            q = (FctInstance * 1)(FctInstance(
                plan.handle.value, *(x.data_ptr() for x in fields),
                (C.c_void_p * 3)(*(b.data_ptr() for b in buf)), ntr, 1200.0, None, None))
            h = C.c_void_p()
            if run == "serve":
                _lib.check(_bind(L).fct_serve_create(0, 1, 1 << 28, C.byref(h)))
                _lib.check(L.fct_serve_step(h, q, (C.c_int32 * 1)(0), 1, s))
            else:
                _lib.check(L.fct_batch_create(q, 1, 1 << 30, C.byref(h)))
                if run == "mapped":
                    _lib.check(L.fct_batch_set_mapping(h, 4, 2))
                _lib.check(L.fct_batch_run(h, 0, 1, s))
            torch.cuda.synchronize()
            got.append(buf[2].clone())
            (L.fct_serve_destroy if run == "serve" else L.fct_batch_destroy)(h)
    assert all(torch.equal(g, got[0]) for g in got)
