"""The network's backward pass after forward passes that did and did not write its transposed activations."""
import numpy as np
import pytest


@pytest.mark.gpu
@pytest.mark.parametrize("rows", [1, 129, 1003])
def test_backward_after_repeated_forward_passes(gpu, rows):
    """A second forward pass without a backward pass between takes the inference route; its backward pass gives the
    gradients of a first one, up to the order of the FP32 atomics (2^-24 of a sum of `rows` products, doubled)."""
    import torch
    from unomol_gb300 import learned
    g = torch.Generator(device="cuda").manual_seed(3)
    x = torch.rand(rows, 20, device="cuda", generator=g)
    dy = torch.rand(rows, 48, device="cuda", generator=g)
    y = torch.empty(rows, 48, device="cuda")
    grads = []
    for passes in (1, 2, 3):
        m = learned.Mlp(20, 64, 3, 48, seed=1)
        for _ in range(passes):
            m.forward(x, y)
        m.backward(dy)
        grads.append(m.grads())
        m.forward(x, y)  # after a backward pass: the training route again
        m.backward(dy)
        grads.append(m.grads())
        m.close()
    for v in grads[1:]:
        assert np.abs(v - grads[0]).max() <= 2.0 * rows * 2.0 ** -24 * np.abs(grads[0]).max()
