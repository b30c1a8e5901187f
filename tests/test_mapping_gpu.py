"""The mapping an ensemble reports is the one its launches take, and the library's choice can
be restored."""

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


def _fields(m, ntr):
    return I.make_fields(m, seed=1, n_passive=max(0, ntr - 2), ab2=True, kind="basin")


def _ensemble(members):
    from fesom_jax_b200.ensemble import Ensemble
    ens = Ensemble()
    for m, ntr in members:
        f = _fields(m, ntr)
        ens.add_member(m, f.uv, f.w_e, f.helem, f.hnode, f.hnode_new, f.tracers[:ntr],
                       f.tracers_old[:ntr], DT)
    ens.build()
    return ens


EVEN = [(2, 1), (2, 1), (2, 1), (2, 2)]
ODD = [(2, 2), (2, 1), (2, 2), (2, 2)]
LARGE = [(4, 1), (4, 1), (4, 1), (2, 2)]


@pytest.mark.gpu
def test_reported_mapping_is_the_one_in_force(torch):
    small, large = (meshgen.make_mesh(n, nl=33, bottom=(3, 33), seed=3) for n in (700, 9000))
    for members, want in (([(small, 2)], EVEN), ([(small, 3)], ODD), ([(large, 8)] * 2, LARGE)):
        ens = _ensemble(members)
        assert ens.stage_map == want == ens.group_mapping(0)
        assert (ens.chunk, ens.levels) == (max(c for c, _ in want), 2)
        ens.run(1)
        ref = ens.state(0)[0].clone()
        ens.set_chunk(1)                     # fewer tracers per thread, the levels stay
        assert ens.stage_map == [(1, lv) for _, lv in want]
        ens.set_mapping(2, 4)
        assert ens.stage_map == [(2, 4)] * 4 and (ens.chunk, ens.levels) == (2, 4)
        ens.set_stage_mapping(1, 1, 8)
        assert ens.stage_map == [(2, 4), (1, 8), (2, 4), (2, 4)]
        ens.reset_mapping()
        assert ens.stage_map == want
        f, ntr = _fields(*members[0]), members[0][1]
        ens.set_state(0, *(torch.from_numpy(x[:ntr]).cuda() for x in (f.tracers, f.tracers_old)))
        ens.run(1)
        assert torch.equal(ens.state(0)[0], ref)
        with pytest.raises(Exception, match="out of range"):
            ens.group_mapping(1)
        ens.close()


@pytest.mark.gpu
def test_groups_keep_their_own_default(torch):
    small = meshgen.make_mesh(700, nl=33, bottom=(3, 33), seed=3)
    ens = _ensemble([(small, 2), (small, 3)])
    assert ens.info()["groups"] == 2
    assert ens.group_mapping(0) == EVEN and ens.group_mapping(1) == ODD
    ens.set_mapping(4, 4)
    assert ens.group_mapping(1) == [(4, 4)] * 4
    ens.reset_mapping()
    assert ens.group_mapping(0) == EVEN and ens.group_mapping(1) == ODD
    ens.close()


@pytest.mark.gpu
def test_autotune_keeps_the_fastest_of_three(torch, tmp_path):
    """The library's choice is timed beside the tuner's, and a cached choice of it is applied
    as the library's choice (each group its own)."""
    from fesom_jax_b200.tuning import TuningCache
    small = meshgen.make_mesh(700, nl=33, bottom=(3, 33), seed=3)
    cache = TuningCache(tmp_path / "tuning.json")
    ens = _ensemble([(small, 2), (small, 3)])
    out = ens.autotune(steps=1, reps=1, cache=cache)
    ms = {"per_stage": out["per_stage_ms"], "uniform": out["uniform_ms"],
          "default": out["default_ms"]}
    assert ms[out["chosen"]] == min(ms.values())
    maps = [ens.group_mapping(g) for g in range(2)]
    again = _ensemble([(small, 2), (small, 3)])
    again.autotune(cache=cache)
    assert [again.group_mapping(g) for g in range(2)] == maps
    key, entry = next(iter(cache._load().items()))
    cache.put(key, {**entry, "chosen": "default"})
    again.set_mapping(1, 8)
    again.autotune(cache=cache)
    assert again.group_mapping(0) == EVEN and again.group_mapping(1) == ODD
    ens.close()
    again.close()
