"""The Python binding's calls: what they accept and refuse, and what they allocate."""
import pytest

from kraken_b200 import capi


@pytest.mark.gpu
def test_silu_mul_keeps_the_layout_of_its_inputs(cuda):
    import torch
    for shape, order in (((64, 32), (1, 0)), ((4, 6, 10), (2, 0, 1))):
        gate, up = (torch.randn(shape, device="cuda").permute(order) for _ in range(2))
        y = cuda.silu_mul(gate, up)
        assert y.stride() == gate.stride() and not y.requires_grad
        want = torch.nn.functional.silu(gate.double()) * up.double()
        assert (y - want).abs().max().item() < 1e-5
