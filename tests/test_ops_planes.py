"""The planes that ops.Context makes for its results (no GPU)."""
import pytest
import torch

from cnet_b200.ops import Context


@pytest.fixture()
def ctx():
    c = object.__new__(Context)
    c.torch, c.h = torch, None
    return c


@pytest.mark.parametrize("make", [lambda: torch.zeros(6, 4).t(), lambda: torch.zeros(4, 12)[:, ::2], lambda: torch.zeros(1, 6).expand(4, 6),
                                  lambda: torch.zeros(4, 6, dtype=torch.float64), lambda: torch.zeros(4, 6, dtype=torch.bfloat16),
                                  lambda: torch.zeros(4, 6, requires_grad=True)])
def test_results_are_contiguous_float32(ctx, make):
    x = make()
    for plane in ctx._like((x, x)):
        assert plane.shape == (4, 6) and plane.dtype == torch.float32 and plane.is_contiguous() and not plane.requires_grad


def test_both_planes_take_the_first_ones_shape(ctx):
    a, b = ctx._like((torch.zeros(4, 6), torch.zeros(6)))
    assert a.shape == b.shape == (4, 6) and a.data_ptr() != b.data_ptr()
