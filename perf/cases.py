"""The measured work of the framework: calls a user's program makes through the public entry
points, over the range of meshes, levels, tracers and options they are made for.

The kinds of work, and what each stands for:

* ``step``: one drop-in ``advect_one_fct`` call, from a few hundred nodes (latency and
  launches) over the pi mesh and a CORE2-size mesh with T and S to a large mesh with several
  tracers; ``options`` adds the moving depths (``Z3d``/``zbar3``) and the split vertical
  velocity (``w_i``).
* ``column``: the tracer part of a model step in its order: ``compute_w``,
  ``advect_one_fct`` of T and S, implicit vertical diffusion with surface forcing and
  shortwave.
* ``ensemble``: resident members advanced by a multi-step graph; ``physics`` adds the w
  producer and the diffusion epilogue, ``tuned`` runs the autotuner first, as the benchmark
  does.
* ``vjp``: forward and backward through the autograd function of the step.
* ``chain``: the loss and gradient of a multi-step run with a kept tape.
* ``ice``: one sea-ice FCT step.

Meshes are the shipped pi mesh and generated ones (``fesom_jax_b200.meshgen``), kept per
process as a program keeps its mesh. Inputs are drawn on the GPU from the seed: profiles
with noise for T and S, uniform passive tracers, closed-basin flows (white noise on pi's
single steps) with w from continuity.
"""

import collections
import math

import numpy as np
import torch

from fesom_jax_b200 import inputs as I
from fesom_jax_b200 import meshgen
from fesom_jax_b200.adjoint import Tape, chain_loss_and_grad, functions
from fesom_jax_b200.ale import compute_w
from fesom_jax_b200.ensemble import Ensemble
from fesom_jax_b200.ice_adv import IceConfig, fct_solve
from fesom_jax_b200.mesh import pi_mesh
from fesom_jax_b200.tracer_adv import advect_one_fct
from fesom_jax_b200.tracer_diff import impl_vert_diff

DEV = "cuda:0"
CORE2 = dict(nodes=127000, nl=48, bottom=5)
PI = dict(nodes=3140, nl=48, bottom=0)   # the shipped mesh (its own bathymetry)


def listed():
    return [
        # the smallest call: one tracer on a coarse test mesh; launches and host time
        dict(name="step_tiny", kind="step", nodes=600, nl=10, bottom=4, ntr=1, options=False),
        # T and S on the shipped pi mesh, the plain single-step configuration
        dict(name="step_pi", kind="step", **PI, ntr=2, options=False),
        # an odd level count and tracer count, with moving depths and split w
        dict(name="step_options", kind="step", nodes=20011, nl=33, bottom=5, ntr=3, options=True),
        # T and S on a CORE2-size mesh: the ordinary model-size call
        dict(name="step_core2", kind="step", **CORE2, ntr=2, options=False),
        # the largest single instance: 70 levels, T and S plus two passive tracers
        dict(name="step_large", kind="step", nodes=300000, nl=70, bottom=10, ntr=4, options=False),
        # the tracer part of a model step at an ordinary size
        dict(name="column_mid", kind="column", nodes=60000, nl=48, bottom=5, ntr=2),
        # many small members: launch-bound graph steps
        dict(name="ensemble_pi", kind="ensemble", **PI, ntr=2, members=16, steps=30,
             physics=False, tuned=False),
        # the batched benchmark's mesh, tracers and mapping search, fewer members
        dict(name="ensemble_core2", kind="ensemble", **CORE2, ntr=8, members=6, steps=6,
             physics=False, tuned=True),
        # odd tracer and member counts with the w producer and the diffusion epilogue
        dict(name="ensemble_physics", kind="ensemble", nodes=30011, nl=40, bottom=5, ntr=5,
             members=3, steps=4, physics=True, tuned=False),
        # forward and backward of one small step
        dict(name="vjp_pi", kind="vjp", **PI, ntr=2),
        # the differentiation benchmark: 10-step loss and gradient
        dict(name="chain_core2", kind="chain", **CORE2, ntr=1, steps=10),
        # sea-ice advection on the CORE2-size surface mesh
        dict(name="ice_core2", kind="ice", **CORE2, ntr=3),
    ]


def draw(rng):
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["step", "step", "column", "ensemble", "ensemble", "vjp", "chain", "ice"])
    nl = rng.randint(10, 70)
    c = dict(kind=kind, nl=nl, bottom=rng.randint(3, max(3, nl // 3)))
    if kind == "step":
        c.update(nodes=size(500, 150000), ntr=rng.randint(1, 4), options=rng.random() < 0.3)
    elif kind == "column":
        c.update(nodes=size(500, 100000), ntr=2)
    elif kind == "ensemble":
        c.update(nodes=size(500, 60000), ntr=rng.choice([1, 2, 3, 4, 5, 6, 8, 10]),
                 members=rng.randint(1, 5), steps=rng.randint(2, 6),
                 physics=rng.random() < 0.3, tuned=False)
    elif kind == "vjp":
        c.update(nodes=size(500, 60000), ntr=rng.randint(1, 3))
    elif kind == "chain":
        c.update(nodes=size(500, 60000), ntr=1, steps=rng.randint(2, 10))
    else:
        c.update(nodes=size(500, 200000), ntr=3)
    return c


# ------------------------------------------------------------------------------- meshes
_meshes = collections.OrderedDict()


def _mesh(case):
    """The case's mesh; the last few are kept, as a program keeps the one it runs on."""
    key = (case["nodes"], case["nl"], case["bottom"])
    if key not in _meshes:
        _meshes[key] = (pi_mesh() if case["bottom"] == 0 else
                        meshgen.make_mesh(case["nodes"], nl=case["nl"],
                                          bottom=(case["bottom"], case["nl"])))
        while len(_meshes) > 4:
            _meshes.popitem(last=False)
    _meshes.move_to_end(key)
    return _meshes[key]


def _host(mesh, name, make):
    """A host array of the mesh that the input generators use again."""
    kept = mesh.__dict__.setdefault("_perf_inputs", {})
    if name not in kept:
        kept[name] = make()
    return kept[name]


def _d(x):
    return torch.as_tensor(np.ascontiguousarray(x), device=DEV)


def _dt(case):
    """A time step that keeps the low-order scheme's Courant number below 1."""
    return 1800.0 * min(1.0, math.sqrt(127000.0 / case["nodes"]))


# ------------------------------------------------------------------------------- inputs
def _gen(seed, salt=0):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed) * 7919 + 104729 * salt + 17)
    return g


def _randn(g, *shape):
    return torch.randn(shape, generator=g, device=DEV, dtype=torch.float64)


def _rand(g, *shape):
    return torch.rand(shape, generator=g, device=DEV, dtype=torch.float64)


def _flow(mesh, g, white):
    """``uv [E, nl, 2]``: closed basins over the bathymetry plus a small divergent part, or
    white noise, with linear decay in the vertical (as ``inputs.basin_velocities``)."""
    decay = _d(1.0 - 0.9 * I.layer_depth_fraction(mesh))
    emask = _d(mesh.elem_layer_mask)
    noise = _randn(g, mesh.elem2D, 2)
    if white:
        return (0.1 * noise[:, None, :] * decay[None, :, None] * emask[:, :, None]).contiguous()
    xyz = _d(I.node_xyz(mesh))
    k = _randn(g, 24, 3)
    k = k / k.norm(dim=1, keepdim=True) * (2.0 + 10.0 * _rand(g, 24, 1))
    psi = (_randn(g, 24) * torch.cos(xyz @ k.T + 2.0 * math.pi * _rand(g, 24))).sum(1)
    gs, en = _d(mesh.gradient_sca), _d(mesh.elem_nodes.astype(np.int64))
    u0 = (gs.view(-1, 2, 3) * psi[en][:, None, :]).sum(2)
    psi = psi * (0.1 / u0.std())
    rings = _host(mesh, "rings", lambda: I.wall_rings(mesh, I.basin_rings(mesh)))
    taper = I.basin_taper([tuple(_d(x) for x in r) for r in rings], mesh.nl, torch)
    psik = psi[:, None] * decay[None, :] * taper
    u, v = torch.zeros_like(emask, dtype=torch.float64), torch.zeros_like(emask, dtype=torch.float64)
    for j in range(3):
        t = psik[en[:, j]]
        u -= gs[:, 3 + j:4 + j] * t
        v += gs[:, j:j + 1] * t
    uv = torch.stack([u, v], 2) + 0.002 * noise[:, None, :] * decay[None, :, None]
    return (uv * emask[:, :, None]).contiguous()


def _tracers(mesh, g, ntr):
    """``T, T_old [ntr, N, nl]``: T, S, then passive tracers; 0 below the bottom."""
    N, nl = mesh.nod2D, mesh.nl
    frac = _d(I.layer_depth_fraction(mesh))[None, :]
    mask = _d(mesh.node_layer_mask)
    T = torch.empty((ntr, N, nl), dtype=torch.float64, device=DEV)
    T_old = torch.empty_like(T)
    for t in range(ntr):
        if t == 0:
            T[t] = 28.0 - 26.0 * frac + 0.5 * _randn(g, N, nl)
        elif t == 1:
            T[t] = 34.0 + 2.0 * frac + 0.1 * _randn(g, N, nl)
        else:
            T[t] = _rand(g, N, nl)
        T[t] *= mask
        T_old[t] = T[t] + 0.05 * _randn(g, N, nl) * mask
    return T, T_old


def _thickness(mesh):
    hn, he = _host(mesh, "rest", lambda: I.rest_thickness(mesh))
    return _d(hn), _d(he)


def _columns(mesh, g):
    """Vertical diffusivity at interfaces: a mixed layer over a weak interior."""
    z = _d(mesh.zbar)[None, :]
    Kv = 1e-5 + 1e-2 * torch.exp(z / 60.0) * (0.5 + _rand(g, mesh.nod2D, mesh.nl))
    return (Kv * _d(mesh.node_iface_mask)).contiguous()


def _fields(case, seed, salt=0):
    mesh, g = _mesh(case), _gen(seed, salt)
    hnode, helem = _thickness(mesh)
    uv = _flow(mesh, g, white=case["bottom"] == 0 and case["kind"] in ("step", "vjp"))
    T, T_old = _tracers(mesh, g, case["ntr"])
    return mesh, g, dict(uv=uv, helem=helem, hnode=hnode, T=T, T_old=T_old)


def prepare(case, seed):
    kind, ntr = case["kind"], case["ntr"]
    if kind == "ensemble":
        ens = Ensemble()
        for i in range(case["members"]):
            mesh, g, f = _fields(case, seed, i)
            ens.add_member(mesh, f["uv"], compute_w(mesh, f["uv"], f["helem"]), f["helem"],
                           f["hnode"], f["hnode"], f["T"], f["T_old"], dt=_dt(case),
                           Kv=_columns(mesh, g) if case["physics"] else None,
                           derive_w=case["physics"])
        ens.build()
        if case["tuned"]:
            ens.autotune()   # it advances the members: put their state back
            for i in range(case["members"]):
                _, _, f = _fields(case, seed, i)
                ens.set_state(i, f["T"], f["T_old"])
        return dict(case=case, ens=ens)
    if kind == "ice":
        mesh, g = _mesh(case), _gen(seed)
        n = mesh.nod2D
        lat = _d(mesh.coord_nod2D[:, 1].copy())
        a = torch.clamp(torch.abs(lat) * 1.2 - 0.6 + 0.1 * _randn(g, n), 0.0, 1.0)
        m = a * (1.0 + _rand(g, n))
        return dict(case=case, mesh=mesh, a=a, m=m, s=0.2 * m * _rand(g, n),
                    u=0.1 * _randn(g, n), v=0.1 * _randn(g, n))
    mesh, g, f = _fields(case, seed)
    s = dict(case=case, mesh=mesh, dt=_dt(case), **f)
    if kind != "chain":
        s["w_e"] = compute_w(mesh, f["uv"], f["helem"])
        if kind in ("step", "vjp") and ntr == 1:
            s["T"], s["T_old"] = f["T"][0].contiguous(), f["T_old"][0].contiguous()
    if kind == "step":
        s["more"] = {}
        if case["options"]:
            zbar, Z = _d(mesh.zbar)[None, :], _d(np.append(mesh.Z, mesh.Z[-1]))[None, :]
            up = 1.0 + 0.01 * _rand(g, mesh.nod2D, 1)   # depths that follow the surface
            s["more"] = dict(Z3d=(Z * up).contiguous(), zbar3=(zbar * up).contiguous(),
                             w_i=(0.3 * s["w_e"]).contiguous())
            s["w_e"] = 0.7 * s["w_e"]
            s["hnode_new"] = s["hnode"] * up
    elif kind == "column":
        s["Kv"] = _columns(mesh, g)
        s["bc"] = 0.01 * _randn(g, ntr, mesh.nod2D)
        s["sw"] = (1e-5 * torch.exp(_d(mesh.zbar)[None, :] / 20.0)
                   * (0.5 + _rand(g, mesh.nod2D, 1))).contiguous()
    elif kind == "vjp":
        for name in ("uv", "w_e", "T", "T_old"):
            s[name].requires_grad_(True)
        s["g"] = _randn(g, *s["T"].shape) * _d(mesh.node_layer_mask)
    elif kind == "chain":
        s["target"] = s["T"][0, :, 0] + 0.1 * _randn(g, mesh.nod2D)
        s["tape"] = Tape(mesh, case["steps"])
    return s


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "step":
        return advect_one_fct(s["mesh"], s["uv"], s["w_e"], s["helem"], s["hnode"],
                              s.get("hnode_new", s["hnode"]), s["T"], s["T_old"], dt=s["dt"],
                              **s["more"])[0]
    if kind == "column":
        m = s["mesh"]
        w = compute_w(m, s["uv"], s["helem"])
        T_new, _ = advect_one_fct(m, s["uv"], w, s["helem"], s["hnode"], s["hnode"], s["T"],
                                  s["T_old"], dt=s["dt"])
        T, S = impl_vert_diff(m, T_new[0], T_new[1], s["Kv"], s["hnode"], dt=s["dt"],
                              bc_T=s["bc"][0], bc_S=s["bc"][1], sw_3d=s["sw"])
        return w, T, S
    if kind == "ensemble":
        s["ens"].run(case["steps"])
        return [s["ens"].state(i) for i in range(case["members"])]
    if kind == "vjp":
        AdvectFCT, _ = functions()
        T_new = AdvectFCT.apply(s["mesh"], s["dt"], s["uv"], s["w_e"], s["helem"], s["hnode"],
                                s["hnode"], s["T"], s["T_old"])
        return (T_new, *torch.autograd.grad(T_new, (s["uv"], s["w_e"], s["T"], s["T_old"]),
                                            s["g"]))
    if kind == "chain":
        return chain_loss_and_grad(s["mesh"], s["T"][0], s["uv"], s["helem"], s["hnode"],
                                   s["hnode"], s["target"], case["steps"], dt=s["dt"],
                                   T_old0=s["T_old"][0], return_gT_old=True, tape=s["tape"])
    return fct_solve(IceConfig(), s["mesh"], s["a"], s["m"], s["s"], s["u"], s["v"])


def work(case):
    """Each input once and each output once: T, T_old and T_new of every wet node level,
    uv and thickness of the wet element levels, w, areas and the mesh; the operations of
    the scheme counted per update (a tracer value at one wet node level)."""
    m = _mesh(case)
    nw, ew, ni = m.n_wet_layers, m.n_wet_elem_layers, m.n_wet_layers + m.nod2D
    mesh2d = 72 * m.edge2D + 96 * m.elem2D + 24 * m.nod2D
    geometry = 8 * ni + 8 * nw + mesh2d
    upd = case["ntr"] * nw
    kind = case["kind"]
    fields = 24 * ew + 8 * ni + 16 * nw   # uv and helem, w, hnode and hnode_new
    if kind == "step":
        more = (16 * ni + 8 * ni) if case["options"] else 0
        return dict(bytes=24 * upd + fields + geometry + more, flops=190 * upd)
    if kind == "column":
        return dict(bytes=24 * upd + fields + geometry + 16 * ni, flops=220 * upd + 25 * nw)
    if kind == "ensemble":
        mem = 24 * upd * case["steps"] + fields + (8 * ni if case["physics"] else 0)
        return dict(bytes=case["members"] * mem + geometry,
                    flops=(220 if case["physics"] else 190) * upd * case["steps"]
                    * case["members"])
    if kind == "vjp":
        return dict(bytes=(24 + 24) * upd + 2 * fields + geometry, flops=700 * upd)
    if kind == "chain":
        return dict(bytes=case["steps"] * (24 + 40) * upd + 2 * fields + geometry,
                    flops=700 * upd * case["steps"])
    return dict(bytes=8 * (3 + 2 + 3) * m.nod2D + 8 * m.nod2D + 68 * m.elem2D,
                flops=1500 * m.nod2D)


def tolerance(case):
    """64-bit throughout. Measured against ``exact``: steps, runs of steps and column solves
    1e-16 to 1.6e-15, gradients 1e-15 to 5e-14 (where two branches of the limiter are within
    rounding of each other another correct implementation may take the other one)."""
    if case["kind"] in ("vjp", "chain"):
        return {"rel": 5e-13, "max": 1e-8}
    return {"rel": 1e-14, "max": 1e-12}


# ------------------------------------------------- the same numbers from plain torch
def _geometry(mesh):
    names = ("edges", "edge_tri", "edge_up_dn_tri", "elem_nodes", "ulevels_nod2D",
             "nlevels_nod2D", "ulevels_nod2D_max", "nlevels_nod2D_min", "ulevels", "nlevels")
    G = {n: _d(np.asarray(getattr(mesh, n)).astype(np.int64)) for n in names}
    for n in ("area", "areasvol", "gradient_sca", "elem_area", "elem_cos", "edge_dxdy",
              "edge_cross_dxdy", "zbar", "Z", "node_layer_mask", "node_iface_mask",
              "elem_layer_mask"):
        G[n] = _d(getattr(mesh, n))
    G["N"], G["nl"] = mesh.nod2D, mesh.nl
    return G


def _down(x):
    return torch.cat([x[..., :1], x[..., :-1]], -1)


def _up(x):
    return torch.cat([x[..., 1:], torch.zeros_like(x[..., :1])], -1)


def _safe(x, bad=1.0):
    return torch.where(x > 0.0, x, torch.full_like(x, bad))


def _nodes(G, vals, ids):
    """Sum of per-entity rows into their nodes."""
    return torch.zeros((G["N"],) + vals.shape[1:], dtype=vals.dtype, device=vals.device) \
        .index_add(0, ids, vals)


def _cell_flux(G, uv, helem):
    """The two cells' volume fluxes through each edge."""
    el1, el2 = G["edge_tri"][:, 0], G["edge_tri"][:, 1]
    e2 = el2.clamp(min=0)
    cr, lm = G["edge_cross_dxdy"], G["elem_layer_mask"]
    U, V = uv[..., 0], uv[..., 1]
    zero = torch.zeros((), dtype=uv.dtype, device=uv.device)
    t1 = torch.where(lm[el1], (U[el1] * cr[:, 1:2] - V[el1] * cr[:, 0:1]) * helem[el1], zero)
    t2 = torch.where(lm[e2] & (el2 >= 0)[:, None],
                     (V[e2] * cr[:, 2:3] - U[e2] * cr[:, 3:4]) * helem[e2], zero)
    return t1, t2


def _exact_w(G, uv, helem):
    t1, t2 = _cell_flux(G, uv, helem)
    c = -(t1 + t2)
    div = _nodes(G, c, G["edges"][:, 0]) - _nodes(G, c, G["edges"][:, 1])
    w = torch.flip(torch.cumsum(torch.flip(div, [1]), 1), [1]) / _safe(G["area"])
    return torch.where(G["node_iface_mask"], w, torch.zeros_like(w))


def _upwind(G, w, T):
    a = w.abs()
    f = -0.5 * (T * (w + a) + _down(T) * (w - a)) * G["area"]
    return torch.where(G["node_layer_mask"], f, torch.zeros_like(f))


def _tdma(a, b, c, d):
    cp, dp = [], []
    cprev = dprev = torch.zeros_like(b[:, 0])
    for k in range(b.shape[1]):
        m = b[:, k] - a[:, k] * cprev
        cprev, dprev = c[:, k] / m, (d[:, k] - a[:, k] * dprev) / m
        cp.append(cprev)
        dp.append(dprev)
    x = [None] * len(cp)
    nxt = torch.zeros_like(cp[0])
    for k in range(len(cp) - 1, -1, -1):
        nxt = dp[k] - cp[k] * nxt
        x[k] = nxt
    return torch.stack(x, 1)


def _exact_step(G, uv, w, helem, hn, hnn, T, T_old, dt, Z3d=None, zbar3=None, w_i=None):
    nlm, ifm, em = G["node_layer_mask"], G["node_iface_mask"], G["elem_layer_mask"]
    n1, n2 = G["edges"][:, 0], G["edges"][:, 1]
    zero = torch.zeros((), dtype=T.dtype, device=T.device)
    k = torch.arange(G["nl"], device=T.device)[None, :]
    top, bot = (G["ulevels_nod2D"] - 1)[:, None], (G["nlevels_nod2D"] - 1)[:, None]
    A = -0.6 * T_old + 1.6 * T
    t1, t2 = _cell_flux(G, uv, helem)
    vf = t1 + t2
    av = vf.abs()
    fl = -0.5 * (T[n1] * (vf + av) + T[n2] * (vf - av))
    fv = _upwind(G, w, T)
    div = _nodes(G, fl, n1) - _nodes(G, fl, n2) + (fv - _up(fv))
    sa, sh = _safe(G["areasvol"]), _safe(hnn)
    valid = nlm & (hnn > 0.0) & (G["areasvol"] > 0.0)
    LO = torch.where(valid, (T * hn + div * dt / sa) / sh, zero)
    if w_i is not None:
        vt, vb = dt * G["area"] / sa, dt * _up(G["area"]) / sa
        wd = _up(w_i)
        lo_b = k == bot - 1
        a = torch.where(k == top, zero, torch.minimum(zero, w_i)) * vt
        bt = torch.where(k == top, w_i, torch.maximum(zero, w_i)) * vt
        bb = torch.where(lo_b, zero, -torch.minimum(zero, wd)) * vb
        c = torch.where(lo_b, zero, -torch.maximum(zero, wd)) * vb
        b = torch.where(nlm, hnn + bt + bb, torch.ones_like(hnn))
        a, c = torch.where(nlm, a, zero), torch.where(nlm, c, zero)
        r = torch.where(nlm, -(a * _down(LO) + (bt + bb) * LO + c * _up(LO)), zero)
        LO = LO + torch.where(nlm, _tdma(a, b, c, r), zero)
        w = w + w_i
        fv = _upwind(G, w, T)
    # MFCT: gradients of the up and down cells, or node averages
    en, gs = G["elem_nodes"], G["gradient_sca"]
    Tv = [T[en[:, j]] for j in range(3)]
    gx = torch.where(em, sum(gs[:, j:j + 1] * Tv[j] for j in range(3)), zero)
    gy = torch.where(em, sum(gs[:, 3 + j:4 + j] * Tv[j] for j in range(3)), zero)
    aw = torch.where(em, G["elem_area"][:, None], zero)
    den = _safe(sum(_nodes(G, aw, en[:, j]) for j in range(3)))
    nx = sum(_nodes(G, gx * aw, en[:, j]) for j in range(3)) / den
    ny = sum(_nodes(G, gy * aw, en[:, j]) for j in range(3)) / den
    up, dn = G["edge_up_dn_tri"][:, 0], G["edge_up_dn_tri"][:, 1]
    lo_k = torch.maximum(G["ulevels_nod2D_max"][n1], G["ulevels_nod2D_max"][n2])[:, None] - 1
    hi_k = torch.minimum(G["nlevels_nod2D_min"][n1], G["nlevels_nod2D_min"][n2])[:, None] - 1
    use = ((up >= 0) & (dn >= 0))[:, None] & (k >= lo_k) & (k < hi_k)
    up, dn = up.clamp(min=0), dn.clamp(min=0)
    R = 6367500.0
    el2 = G["edge_tri"][:, 1]
    a = R * G["elem_cos"][G["edge_tri"][:, 0]]
    a = torch.where(el2 >= 0, 0.5 * (a + R * G["elem_cos"][el2.clamp(min=0)]), a)[:, None]
    ex, ey = G["edge_dxdy"][:, 0:1] * a, G["edge_dxdy"][:, 1:2] * R
    d = A[n2] - A[n1]
    Tm1 = A[n1] + (2.0 * d + ex * torch.where(use, gx[up], nx[n1])
                   + ey * torch.where(use, gy[up], ny[n1])) / 6.0
    Tm2 = A[n2] - (2.0 * d + ex * torch.where(use, gx[dn], nx[n2])
                   + ey * torch.where(use, gy[dn], ny[n2])) / 6.0
    ah = -0.5 * ((vf + av) * Tm1 + (vf - av) * Tm2) - fl
    # QR4C
    if Z3d is None:
        Zp = torch.cat([G["Z"], G["Z"][-1:]])[None, :]
        zb = G["zbar"][None, :]
    else:
        Zp, zb = Z3d, zbar3
    Zm1 = _down(Zp)
    Zm2, Zn = _down(Zm1), torch.cat([Zp[:, 1:], Zp[:, -1:]], 1)

    def gap(x):
        return torch.where(x == 0.0, torch.ones_like(x), x)

    Am1, Ap1 = _down(A), _up(A)
    Am2 = _down(Am1)
    qc, qu, qd = (Am1 - A) / gap(Zm1 - Zp), (A - Ap1) / gap(Zp - Zn), (Am2 - Am1) / gap(Zm2 - Zm1)
    m1 = A + (2.0 * qc + qu) * (zb - Zp) / 3.0
    m2 = Am1 + (2.0 * qc + qd) * (zb - Zm1) / 3.0
    wa = w * G["area"]
    hi = torch.where((k >= top + 2) & (k <= bot - 2), -0.5 * (m1 + m2) * wa, zero)
    hi = torch.where((k == top + 1) | (k == bot - 1), -0.5 * (Am1 + A) * wa, hi)
    hi = torch.where(k == bot, zero, hi)
    hi = torch.where(k == top, -A * wa, hi)
    av_ = torch.where(ifm, hi, zero) - fv
    # Zalesak
    big = torch.full((), 1e3, dtype=T.dtype, device=T.device)
    tx, tn = torch.maximum(LO, T), torch.minimum(LO, T)
    ax = torch.where(em, torch.amax(torch.stack([tx[en[:, j]] for j in range(3)]), 0), -big)
    an = torch.where(em, torch.amin(torch.stack([tn[en[:, j]] for j in range(3)]), 0), big)
    seg = en.T.reshape(-1)[:, None].expand(-1, G["nl"])
    vx = torch.zeros_like(T).scatter_reduce(0, seg, ax.repeat(3, 1), "amax", include_self=False)
    vn = torch.zeros_like(T).scatter_reduce(0, seg, an.repeat(3, 1), "amin", include_self=False)
    own = (k == top) | (k == bot - 1)
    wx = torch.where(own, vx, torch.maximum(torch.maximum(_down(vx), vx), _up(vx)))
    wn = torch.where(own, vn, torch.minimum(torch.minimum(_down(vn), vn), _up(vn)))
    wx, wn = torch.where(nlm, wx - LO, zero), torch.where(nlm, wn - LO, zero)
    fb = _up(av_)
    plus = torch.where(nlm, torch.maximum(av_, zero) + torch.maximum(-fb, zero), zero) \
        + _nodes(G, torch.maximum(ah, zero), n1) + _nodes(G, torch.maximum(-ah, zero), n2)
    minus = torch.where(nlm, torch.minimum(av_, zero) + torch.minimum(-fb, zero), zero) \
        + _nodes(G, torch.minimum(ah, zero), n1) + _nodes(G, torch.minimum(-ah, zero), n2)
    one = torch.ones((), dtype=T.dtype, device=T.device)
    pf = torch.where(valid, torch.minimum(one, wx / (plus * dt / sa / sh + 1e-16)), one)
    mf = torch.where(valid, torch.minimum(one, wn / (minus * dt / sa / sh - 1e-16)), one)
    ae = torch.where(av_ >= 0.0, torch.minimum(_down(mf), pf), torch.minimum(_down(pf), mf))
    ae = torch.where(k == top, torch.where(av_ >= 0.0, pf, mf), ae)
    lv = torch.where(ifm, ae * av_, zero)
    lh = torch.where(ah >= 0.0, torch.minimum(pf[n1], mf[n2]), torch.minimum(mf[n1], pf[n2])) * ah
    hs = _nodes(G, lh, n1) - _nodes(G, lh, n2)
    vd = torch.where(G["areasvol"] > 0.0, (lv - _up(lv)) * dt / sa, zero)
    dT = torch.where(nlm, -T * hn + LO * hnn + vd, zero) + torch.where(nlm, hs * dt / sa, zero)
    dT = dT + T * (hn - hnn)
    return T + torch.where(nlm & (hnn > 0.0), dT / sh, zero)


def _exact_diffusion(G, T, Kv, hnn, dt, bc=None, sw=None):
    nlm = G["node_layer_mask"]
    k = torch.arange(G["nl"], device=T.device)[None, :]
    top, bot = (G["ulevels_nod2D"] - 1)[:, None], (G["nlevels_nod2D"] - 1)[:, None]
    Zp = torch.cat([G["Z"], G["Z"][-1:]])[None, :]
    du, dd = _down(Zp) - Zp, Zp - _up(Zp)
    du, dd = torch.where(du == 0.0, 1.0, du), torch.where(dd == 0.0, 1.0, dd)
    sa = _safe(G["areasvol"])
    zero = torch.zeros((), dtype=T.dtype, device=T.device)
    a = torch.where(nlm & (k != top), -Kv * dt / du * (G["area"] / sa), zero)
    c = torch.where(nlm & (k != bot - 1), -_up(Kv) * dt / dd * (_up(G["area"]) / sa), zero)
    b = torch.where(nlm, hnn - a - c, torch.ones_like(hnn))
    r = torch.where(nlm, a * (T - _down(T)) + c * (T - _up(T)), zero)
    if bc is not None:
        r = r + torch.where((k == top) & nlm, bc[:, None], zero)
    if sw is not None:
        r = r + torch.where(nlm, (sw - _up(sw) * (_up(G["area"]) / sa)) * dt, zero)
    return T + torch.where(nlm, _tdma(a, b, c, r), zero)


def _exact_ice(G, s):
    en, vol = G["elem_nodes"], G["elem_area"]
    dx, dy = G["gradient_sca"][:, 0:3], G["gradient_sca"][:, 3:6]
    cfg = IceConfig()
    dt, gamma = cfg.ice_dt, cfg.ice_gamma_fct
    ia = 1.0 / _safe(G["area"][:, 0])
    ice_e, ice_n = (G["ulevels"] <= 1)[:, None], G["ulevels_nod2D"] <= 1
    zero = torch.zeros((), dtype=vol.dtype, device=vol.device)

    def gather(c):
        return _nodes(G, torch.where(ice_e, c, zero).reshape(-1), en.reshape(-1))

    def mass(x):
        xv = x[en]
        return gather((vol / 12.0)[:, None] * (xv + xv.sum(1, keepdim=True)))

    U, V = s["u"][en], s["v"][en]
    um, vm = U.sum(1), V.sum(1)
    diff = cfg.ice_diff * torch.sqrt(vol / 2.0e8)
    a = (dx[:, :, None] * (um[:, None, None] + U[:, None, :])
         + dy[:, :, None] * (vm[:, None, None] + V[:, None, :])) / 12.0
    b = diff[:, None, None] * (dx[:, :, None] * dx[:, None, :] + dy[:, :, None] * dy[:, None, :])
    ud = um[:, None] * dx + vm[:, None] * dy
    E = vol[:, None, None] * dt * (a - b - 0.5 * dt * (ud[:, :, None] * ud[:, None, :]) / 9.0)
    out = []
    for X in (s["a"], s["m"], s["s"]):
        rhs = gather((E * X[en][:, None, :]).sum(2))
        d = torch.where(ice_n, rhs * ia, zero)
        for _ in range(2):
            d = torch.where(ice_n, d + (rhs - mass(d)) * ia, d)
        lo = torch.where(ice_n, (rhs + gamma * mass(X)) * ia + (1.0 - gamma) * X, X)
        wv = (gamma * X + d)[en]
        f = -(wv.sum(1, keepdim=True) - 3.0 * wv) * (vol[:, None] * ia[en]) / 12.0
        f = torch.where(ice_e, f, zero)
        inf = torch.full((), math.inf, dtype=vol.dtype, device=vol.device)
        hi_e = torch.where(ice_e[:, 0], torch.maximum(lo[en].amax(1), X[en].amax(1)), -inf)
        lo_e = torch.where(ice_e[:, 0], torch.minimum(lo[en].amin(1), X[en].amin(1)), inf)
        seg = en.reshape(-1)
        hi = torch.full_like(X, -math.inf).scatter_reduce(0, seg, hi_e.repeat_interleave(3), "amax")
        low = torch.full_like(X, math.inf).scatter_reduce(0, seg, lo_e.repeat_interleave(3), "amin")
        hi = torch.where(torch.isfinite(hi), hi, zero) - lo
        low = torch.where(torch.isfinite(low), low, zero) - lo
        fp, fm = gather(torch.maximum(f, zero)), gather(torch.minimum(f, zero))
        pp = torch.where(fp > 0.0, torch.clamp(hi / fp.clamp(min=1e-12), max=1.0), zero)
        pm = torch.where(fm < 0.0, torch.clamp(low / fm.clamp(max=-1e-12), max=1.0), zero)
        pp, pm = torch.where(ice_n, pp, zero), torch.where(ice_n, pm, zero)
        ae = torch.where(f >= 0.0, pp[en], pm[en]).amin(1, keepdim=True)
        out.append(lo + gather(f * ae))
    return tuple(out)


def exact(case, seed):
    kind = case["kind"]
    G = _geometry(_mesh(case))
    if kind == "ensemble":
        if case["nodes"] * case["nl"] * case["ntr"] * case["members"] * case["steps"] > 3e9:
            return None
        out = []
        for i in range(case["members"]):
            mesh, g, f = _fields(case, seed, i)
            w = _exact_w(G, f["uv"], f["helem"])
            Kv = _columns(mesh, g) if case["physics"] else None
            T, T_old = f["T"].clone(), f["T_old"].clone()
            for t in range(case["ntr"]):
                for _ in range(case["steps"]):
                    new = _exact_step(G, f["uv"], w, f["helem"], f["hnode"], f["hnode"], T[t],
                                      T_old[t], _dt(case))
                    if Kv is not None:
                        new = _exact_diffusion(G, new, Kv, f["hnode"], _dt(case))
                    T_old[t] = T[t]
                    T[t] = new
            out.append((T, T_old))
        return out
    s = prepare(case, seed)
    if kind == "ice":
        return _exact_ice(G, s)
    uv, helem, hn, dt = s["uv"], s["helem"], s["hnode"], s["dt"]
    T = s["T"] if s["T"].dim() == 3 else s["T"][None]
    T_old = s["T_old"] if s["T"].dim() == 3 else s["T_old"][None]
    if kind == "step":
        new = torch.stack([_exact_step(G, uv, s["w_e"], helem, hn, s.get("hnode_new", hn), T[t],
                                       T_old[t], dt, **s["more"]) for t in range(case["ntr"])])
        return new if s["T"].dim() == 3 else new[0]
    if kind == "column":
        w = _exact_w(G, uv, helem)
        new = [_exact_diffusion(G, _exact_step(G, uv, w, helem, hn, hn, T[t], T_old[t], dt),
                                s["Kv"], hn, dt, s["bc"][t], s["sw"] if t == 0 else None)
               for t in range(2)]
        return (w, *new)
    if kind == "vjp":
        x = [s[n] for n in ("uv", "w_e", "T", "T_old")]
        new = torch.stack([_exact_step(G, x[0], x[1], helem, hn, hn, T[t], T_old[t], dt)
                           for t in range(case["ntr"])])
        new = new if s["T"].dim() == 3 else new[0]
        return (new, *torch.autograd.grad(new, x, s["g"]))
    from torch.utils.checkpoint import checkpoint
    uv, T0, To0 = (x.detach().requires_grad_(True) for x in (uv, T[0], T_old[0]))
    w = _exact_w(G, uv, helem)
    T, T_old = T0, To0
    for _ in range(case["steps"]):
        T, T_old = checkpoint(_exact_step, G, uv, w, helem, hn, hn, T, T_old, dt,
                              use_reentrant=False), T
    loss = (G["areasvol"][:, 0] * (T[:, 0] - s["target"]) ** 2).sum()
    gT, guv, gTo = torch.autograd.grad(loss, (T0, uv, To0))
    return float(loss.detach()), gT, guv, gTo
