"""The surrogate's whole passes (one launch per layer) against its layer-by-layer
passes: the same bits for predictions, gradients and Adam steps, over ragged
batches, widths off the tile sizes, split-K sums inside a CTA and across CTAs,
tall and short bias sums, and networks the whole passes leave to the others."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _layers(name):
    from ionosphere_fdtd_b200.surrogate import Layer, architecture

    return {
        "default": architecture(),
        "narrow": architecture(width=136, depth=3),
        "two_decoders": architecture(width=256, depth=2, t0=64, c0=32, channels=(16, 1)),
        "one_wide": [Layer(64, 2048, 1, 1), Layer(2048, 520, 1, 1), Layer(520, 16, 1, 1)],
        "small": [Layer(8, 24, 1, 3), Layer(8, 16, 0, 1)],
        "odd_outputs": [Layer(16, 8, 1, 1), Layer(8, 7, 0, 1)],
    }[name]


def _pair(name, seed=0):
    from ionosphere_fdtd_b200.surrogate import TraceSurrogate

    return TraceSurrogate(_layers(name), seed=seed), TraceSurrogate(_layers(name), seed=seed)


def _inputs(layers, batch):
    import torch

    g = torch.Generator(device="cuda").manual_seed(batch)
    x = (2.0 * torch.rand((batch, layers[0].fan_in), generator=g, device="cuda") - 1.0).to(torch.bfloat16)
    return x, g


def _status():
    from ionosphere_fdtd_b200 import _native as N

    out = N.C.c_int32(-1)
    N.check(N.load().ifdtd_nn_gemm_tc_status(1, N.C.byref(out)), "ifdtd_nn_gemm_tc_status")
    return out.value


@pytest.mark.parametrize("name,batch", [("default", 1), ("default", 300), ("default", 512), ("narrow", 77), ("two_decoders", 129),
                                        ("one_wide", 512), ("small", 200), ("small", 5000), ("odd_outputs", 4200)])
def test_whole_pass_equals_layer_by_layer(name, batch):
    import torch

    from ionosphere_fdtd_b200 import _native as N

    whole, single = _pair(name)
    x, g = _inputs(whole.layers, batch)
    for step in range(2):
        p, q = whole.forward(x), single._forward_layers(x)
        assert whole._pass is not None and torch.equal(p, q)
        for (xa, za), (xb, zb) in zip(whole._acts, single._acts):
            assert torch.equal(xa, xb) and torch.equal(za, zb)
        grad = torch.randn(p.shape, generator=g, device="cuda")
        assert whole._backward_whole(grad)
        single._backward_layers(grad)
        for i in range(len(whole.layers)):
            assert torch.equal(whole.gw[i], single.gw[i]), ("gw", i)
            assert torch.equal(whole.gb[i], single.gb[i]), ("gb", i)
        whole.adam_step(1e-3)
        single.step_count += 1
        for w, gr, m, v, w16 in [*zip(single.w, single.gw, single.mw, single.vw, single.w16),
                                 *zip(single.b, single.gb, single.mb, single.vb, [None] * len(single.b))]:
            N.check(N.load().ifdtd_nn_adam(w.numel(), w.data_ptr(), gr.data_ptr(), m.data_ptr(), v.data_ptr(), 1e-3, 0.9, 0.999, 1e-8,
                                           single.step_count, None if w16 is None else w16.data_ptr(), single._stream()), "ifdtd_nn_adam")
        for a, b in zip(whole.w + whole.b + whole.w16 + whole.mw + whole.vb, single.w + single.b + single.w16 + single.mw + single.vb):
            assert torch.equal(a, b)
    assert _status() == 0


@pytest.mark.parametrize("cases,batch", [(1, 512), (512, 512), (513, 512), (1000, 300), (5000, 512), (700, 7)])
def test_grouped_prediction_equals_batches(cases, batch):
    import torch

    whole, single = _pair("narrow", seed=4)
    x, _ = _inputs(whole.layers, cases)
    ref = torch.cat([single._forward_layers(x[i : i + batch].contiguous()).clone() for i in range(0, cases, batch)])
    assert torch.equal(whole.predict(x, batch=batch), ref)
    # the activations kept are the last batch's, as after a forward pass on it
    assert int(whole._acts[0][0].shape[0]) == cases - (cases - 1) // batch * batch
    with pytest.raises((RuntimeError, ValueError)):
        whole.predict(x[:0])
    assert _status() == 0


def test_networks_outside_the_whole_pass():
    """A fan-in that is no multiple of eight, the mma.sync product and an unaligned
    input run layer by layer, and gradients may be replaced before a step."""

    import torch

    from ionosphere_fdtd_b200.surrogate import Layer, TraceSurrogate

    odd = TraceSurrogate([Layer(8, 12, 1, 1), Layer(12, 4, 0, 1)], seed=1)
    x, g = _inputs(odd.layers, 33)
    p = odd.forward(x)
    odd.backward(torch.ones_like(p))
    odd.adam_step(1e-3)
    assert odd._pass is None and np.isfinite(odd.w[0].cpu().numpy()).all()
    net, ref = _pair("small")
    shifted = torch.empty(65 * 8 + 1, dtype=torch.bfloat16, device="cuda")[1:].view(65, 8)
    shifted.copy_(_inputs(net.layers, 65)[0])
    assert torch.equal(net.forward(shifted), ref._forward_layers(shifted.clone())) and net._pass is None
    assert TraceSurrogate(net.layers, seed=0, gemm="mma").forward(x).shape == (33, 48)
    pred = ref.forward(x)
    ref.backward(torch.ones_like(pred))
    ref.gw = [torch.zeros_like(w) for w in ref.gw]
    before = ref.w[0].clone()
    ref.adam_step(1e-2)
    assert torch.equal(ref.w[0], before) and not torch.equal(ref.b[0], torch.zeros_like(ref.b[0]))
