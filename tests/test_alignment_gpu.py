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
