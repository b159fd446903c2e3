"""The medium the misfit hands to a session: interleaved and padded exactly as
numpy's edge padding does, without device memory of its own (torch would keep
it while the gradient sizes its stores from what is free)."""

import numpy as np
import pytest
import torch

from cgfdm import autograd


def _oracle(vp, vs, rho):
    m = np.stack([np.asarray(t.detach().cpu(), np.float32) for t in (vs, vp, rho)], axis=-1)
    return np.pad(m, ((3, 3), (3, 3), (3, 3), (0, 0)), mode="edge")


def _fields(shape, device, dtype=torch.float32):
    g = torch.Generator().manual_seed(sum(shape))
    return [torch.rand(shape, generator=g, dtype=torch.float64).to(device, dtype).requires_grad_() for _ in range(3)]


@pytest.mark.parametrize("shape", [(1, 1, 1), (1, 4, 2), (2, 1, 7), (5, 6, 7), (33, 17, 40)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.float64, torch.float16])
def test_padded_medium_is_edge_padding(shape, dtype):
    vp, vs, rho = _fields(shape, "cpu", dtype)
    for args in ((vp, vs, rho), (vp.transpose(0, 2), vs.transpose(0, 2), rho.transpose(0, 2)),
                 (vp, vs.expand(shape), torch.flip(rho, (0, 1)))):
        got = autograd._padded_medium(*args)
        assert got.dtype == np.float32 and got.flags.c_contiguous
        np.testing.assert_array_equal(got, _oracle(*args))


def test_padded_medium_is_made_on_the_host_whatever_the_default_device():
    vp, vs, rho = _fields((3, 4, 5), "cpu")
    with torch.device("meta"):
        got = autograd._padded_medium(vp, vs, rho)
    np.testing.assert_array_equal(got, _oracle(vp, vs, rho))


@pytest.mark.parametrize("shapes", [((4, 4, 4), (4, 4, 4), (4, 4, 5)), ((4, 4), (4, 4), (4, 4))])
def test_padded_medium_refuses_other_shapes(shapes):
    with pytest.raises(ValueError):
        autograd._padded_medium(*[torch.ones(s) for s in shapes])


@pytest.mark.gpu
@pytest.mark.parametrize("shape", [(104, 136, 144), (33, 17, 40)])
def test_padded_medium_takes_no_device_memory(shape):
    vp, vs, rho = _fields(shape, "cuda")
    want = _oracle(vp, vs, rho)
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    torch.cuda.reset_peak_memory_stats()
    before, reserved = torch.cuda.memory_allocated(), torch.cuda.memory_reserved()
    got = autograd._padded_medium(vp, vs, rho)
    assert torch.cuda.max_memory_allocated() == before and torch.cuda.memory_reserved() == reserved
    np.testing.assert_array_equal(got, want)
