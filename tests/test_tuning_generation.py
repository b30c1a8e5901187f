"""A tuning entry belongs to the kernels it was timed on: one that other kernels wrote (with
another generation in its key, or none) is not applied."""

from fesom_jax_b200 import tuning
from fesom_jax_b200.mesh import pi_mesh


def test_entries_of_other_kernels_are_passed_over(tmp_path, monkeypatch):
    m = pi_mesh()
    cache = tuning.TuningCache(tmp_path / "tuning.json")
    shape = dict(members=32, ntr=8)
    # as the first kernels' autotuner wrote it
    cache.put(f"ensemble|NVIDIA B200|{tuning.mesh_fingerprint(m)}|members=32,ntr=8",
              {"stage_map": [[2, 4]] * 4})
    assert cache.get(tuning.key("ensemble", "NVIDIA B200", [m], **shape)) is None
    mine = tuning.key("ensemble", "NVIDIA B200", [m], **shape)
    cache.put(mine, {"stage_map": [[4, 1]] * 4})
    monkeypatch.setattr(tuning, "KERNELS", tuning.KERNELS + 1)
    assert cache.get(tuning.key("ensemble", "NVIDIA B200", [m], **shape)) is None
    monkeypatch.undo()
    assert cache.get(tuning.key("ensemble", "NVIDIA B200", [m], **shape)) == \
        {"stage_map": [[4, 1]] * 4}
