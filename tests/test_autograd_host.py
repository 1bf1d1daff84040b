"""Host logic of the differentiable exchange that needs no GPU."""
import itertools

import pytest
import torch

from ghex_b200.autograd import _dense


@pytest.mark.parametrize("shape", [(2, 3, 5), (1, 4, 3), (1, 1, 1), (4, 1, 2)])
def test_dense_is_what_empty_like_keeps(shape):
    t = torch.empty(4096)
    for order, gap in itertools.product(itertools.permutations(range(3)), (0, 1)):
        stride, n = [0] * 3, 1
        for d in order:
            stride[d] = n
            n *= shape[d] + gap
        v = t.as_strided(shape, stride)
        assert _dense(v.shape, v.stride()) == (torch.empty_like(v).stride() == v.stride())
    assert not _dense((2, 2), (0, 1))
