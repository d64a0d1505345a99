"""The rows that the surrogate network makes of its inputs and targets: every shape that an assignment to an (n, width) array
takes, and no other. No GPU needed."""

from __future__ import annotations

import numpy as np
import pytest

from wadi2d_b200.surrogate import Network


def _network():
    import torch

    net = object.__new__(Network)
    net.torch, net.device = torch, torch.device("cpu")
    return net


@pytest.mark.parametrize("n", [1, 5, 16])
@pytest.mark.parametrize("shape", [(), (1,), (16,), (5,), (5, 1), (1, 16), (5, 16), (16, 16), (1, 5, 16), (1, 1, 16), (1, 1, 1),
                                   (2, 5, 16), (5, 1, 16), (1, 1, 5, 16), (1, 5, 1)])  # fmt: skip
@pytest.mark.parametrize("dtype", [np.float32, np.float64, np.int64])
def test_rows_are_what_an_assignment_gives(shape, n, dtype):
    import torch

    net = _network()
    x = np.random.default_rng(1).integers(-9, 9, shape).astype(dtype)
    want = torch.zeros((n, 16))
    try:
        want[:n] = torch.as_tensor(np.asarray(x, np.float32))
    except RuntimeError:
        with pytest.raises(RuntimeError):
            net._rows(x, 16, n)
        return
    got, rows = net._rows(x, 16, n)
    assert rows == n and got.is_contiguous() and got.dtype == torch.float32 and got.data_ptr() % 16 == 0
    assert torch.equal(got, want)
