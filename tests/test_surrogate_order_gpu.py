"""Layer launches that follow each other while their CTAs wait for tensor memory.

In a pass of a few thousand cases a launch has more CTAs of 64 to 256 columns than
the SMs' tensor memory holds at once, so CTAs of one launch wait for columns while
the next launch is allowed to begin: the results are the layer-by-layer ones, and
every pass ends.
"""

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", [1024, 3584, 4095])
def test_launches_short_of_tensor_memory(rows):
    import torch

    from ionosphere_fdtd_b200.surrogate import TraceSurrogate, architecture

    net, ref = TraceSurrogate(architecture(), seed=2), TraceSurrogate(architecture(), seed=2)
    g = torch.Generator(device="cuda").manual_seed(rows)
    x = (2.0 * torch.rand((rows, 8), generator=g, device="cuda") - 1.0).to(torch.bfloat16)
    expected = ref._forward_layers(x)
    grad = torch.randn(expected.shape, generator=g, device="cuda")
    ref._backward_layers(grad)
    for _ in range(20):
        out = net.forward(x)
        net.backward(grad)
    assert net._pass is not None and torch.equal(out, expected)
    for a, b in zip(net.gw + net.gb, ref.gw + ref.gb):
        assert torch.equal(a, b)
    torch.cuda.synchronize()
