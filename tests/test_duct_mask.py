"""duct_mask over the forms an obstacle can come in, on the CPU: the mask is a plain C-ordered
byte array, 1 where the obstacle is not 0, with the walls (1|8) over it."""
import numpy as np
import pytest

from myfluidsimulation_b200 import workloads as W

DIMS = (6, 5, 4)
HIT = np.random.default_rng(0).random(DIMS[::-1]) < 0.3


def as_tensor(a):
    import torch
    return torch.tensor(a)


@pytest.mark.parametrize("form", [
    lambda h: h, lambda h: h.astype(np.uint8) * 7, lambda h: np.where(h, np.nan, 0.0), lambda h: h.astype(object),
    lambda h: h.ravel(), np.asfortranarray, lambda h: h[:, ::-1][:, ::-1], lambda h: np.ma.masked_array(h, mask=h), as_tensor,
    lambda h: as_tensor(h.astype(np.float32)).requires_grad_(),
], ids=["bool", "uint8", "float", "object", "flat", "fortran", "strided", "masked", "torch", "torch-grad"])
def test_mask_of_every_form_of_obstacle(form):
    nx, ny, nz = DIMS
    want = np.zeros((nz, ny, nx), np.uint8)
    want[HIT] = 1
    want[:, [0, -1], :] = want[[0, -1]] = W.MASK_SOLID | W.MASK_WALL
    h = HIT.copy()
    got = W.duct_mask(nx, ny, nz, form(h))
    assert type(got) is np.ndarray and got.dtype == np.uint8 and got.flags.c_contiguous and got.flags.writeable
    np.testing.assert_array_equal(got, want)
    np.testing.assert_array_equal(h, HIT)
