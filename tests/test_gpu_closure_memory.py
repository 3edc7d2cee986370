"""The closure keeps device copies of the arrays its calls take from the host, and
only of those: a forward pass has no target."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_a_forward_pass_keeps_its_input_only():
    import torch
    from lbman3d_b200.closure import Closure
    V = 128 ** 3
    with Closure(128, 128, 128, seed=1) as c:
        x = np.zeros((9, V), np.float32)
        torch.cuda.synchronize()
        free = torch.cuda.mem_get_info()[0]
        c.forward(x)
        torch.cuda.synchronize()
        assert free - torch.cuda.mem_get_info()[0] <= 4 * 9 * V + (8 << 20)  # the target's 8 V floats are 64 MB
