"""What the surrogate's whole passes refuse before any device work, and what they
leave to the layer-by-layer passes (no device: the addresses are never used)."""

import ctypes as C
import threading
from types import SimpleNamespace

import pytest

from ionosphere_fdtd_b200 import _native as N
from ionosphere_fdtd_b200 import surrogate
from ionosphere_fdtd_b200.surrogate import Layer, TraceSurrogate, architecture

BASE = 1 << 40


def _layers(shapes):
    """Descriptors whose arrays lie at made-up 256-byte aligned addresses."""

    net = (N.NetLayer * len(shapes))()
    at = BASE
    for d, (fan_in, fan_out, act, expand) in zip(net, shapes):
        d.fan_in, d.fan_out, d.act, d.expand = fan_in, fan_out, act, expand
        for name in ("w16", "bias", "z", "y", "dz", "dz16", "gw", "gb"):
            setattr(d, name, at)
            at += 1 << 36
    return net


SHAPES = [(8, 64, 1, 4), (16, 4, 0, 1)]


@pytest.mark.parametrize("rows", [1 << 25, 1 << 26])
def test_layers_of_2_to_the_31_values_are_left_to_the_separate_kernels(rows):
    assert N.load().ifdtd_nn_forward(_layers(SHAPES), 2, rows, rows, BASE, None) == N.ERR_UNSUPPORTED
    net = object.__new__(TraceSurrogate)
    net.gemm_entry, net.layers = "ifdtd_nn_gemm_tc_ws", [Layer(*s) for s in SHAPES]
    x = SimpleNamespace(shape=(rows, 8), data_ptr=lambda: BASE)
    assert not net._whole_pass(x)
    x.shape = ((1 << 25) - 1, 8)
    assert net._whole_pass(x)
    net.layers = architecture()
    x.shape = (524_288, 8)
    assert not net._whole_pass(x)


@pytest.mark.parametrize("name", ["gw", "dz", "dz16", "z", "y", "w16"])
def test_unaligned_arrays_are_refused_before_a_launch(name):
    lib, rows, need = N.load(), 300, C.c_int64()
    net = _layers(SHAPES)
    assert lib.ifdtd_nn_backward_bytes(net, 2, rows, C.byref(need)) == N.OK
    setattr(net[0], name, getattr(net[0], name) + 4)
    args = (BASE, BASE, BASE, BASE, need.value, None)
    assert lib.ifdtd_nn_backward(net, 2, rows, *args) == N.ERR_UNSUPPORTED
    if name in ("z", "y", "w16"):
        assert lib.ifdtd_nn_forward(net, 2, rows, rows, BASE, None) == N.ERR_UNSUPPORTED


def test_an_unaligned_gradient_is_refused_before_a_launch():
    lib, rows, need = N.load(), 300, C.c_int64()
    net = _layers(SHAPES)
    assert lib.ifdtd_nn_backward_bytes(net, 2, rows, C.byref(need)) == N.OK
    assert lib.ifdtd_nn_backward(net, 2, rows, BASE, BASE + 4, BASE, BASE, need.value, None) == N.ERR_UNSUPPORTED


def _hostless(monkeypatch, forward, shapes):
    """A model on host tensors whose forward launches are ``forward``."""

    import torch

    monkeypatch.setattr(surrogate, "_lib", lambda: SimpleNamespace(
        ifdtd_nn_forward=forward, ifdtd_nn_backward_bytes=N.load().ifdtd_nn_backward_bytes))
    monkeypatch.setattr(TraceSurrogate, "_stream", lambda self: None)
    model = object.__new__(TraceSurrogate)
    model.torch, model.device, model.gemm_entry = torch, torch.device("cpu"), "ifdtd_nn_gemm_tc_ws"
    model.layers, model._layout = [Layer(*s) for s in shapes], None
    model.w16 = [torch.zeros((L.fan_out, L.fan_in), dtype=torch.bfloat16) for L in model.layers]
    model.b = [torch.zeros(L.fan_out) for L in model.layers]
    return model


@pytest.mark.parametrize("infer", [False, True])
def test_passes_of_two_threads_keep_their_own_arrays(monkeypatch, infer):
    """Both threads have described their pass before either is enqueued."""

    import torch

    met, enqueued = threading.Barrier(2, timeout=30), {}

    def forward(net, n, rows, rows_per_pass, x, stream):
        met.wait()
        enqueued[x] = (rows, net[n - 1].z)
        return N.OK

    model = _hostless(monkeypatch, forward, SHAPES)
    xs = [torch.zeros((rows, 8), dtype=torch.bfloat16) for rows in (24, 40)]
    outs = [torch.zeros((len(x), 16)) for x in xs]
    run = (lambda x, o: model._infer(x, len(x), o)) if infer else model._forward
    threads = [threading.Thread(target=run, args=a) for a in zip(xs, outs)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert enqueued == {x.data_ptr(): (len(x), o.data_ptr()) for x, o in zip(xs, outs)}


@pytest.mark.parametrize("cases", [16, 40, 100])
def test_a_prediction_is_not_the_kept_activations(monkeypatch, cases):
    """A program may overwrite its predictions before it asks for gradients."""

    import torch

    def forward(net, n, rows, rows_per_pass, x, stream):
        C.memset(net[n - 1].z, 0, rows * 16 * 4)
        return N.OK

    model = _hostless(monkeypatch, forward, SHAPES)
    out = model.predict(torch.zeros((cases, 8), dtype=torch.bfloat16), batch=16)
    assert out.shape == (cases, 16) and not out.any()
    out.fill_(7.0)
    assert not model._acts[-1][1].any()


def test_grouped_batches_are_bounded_in_memory(monkeypatch):
    """The caller's batch bounds a prediction's memory: several batches share a pass
    only while their activations stay small."""

    import torch

    rows = []

    def forward(net, n, count, rows_per_pass, x, stream):
        rows.append(count)
        return N.OK

    wide = 1 << 20  # 2 MiB of activations per case
    model = _hostless(monkeypatch, forward, [(8, wide, 1, wide // 8), (8, 1, 0, 1)])
    model.predict(torch.zeros((300, 8), dtype=torch.bfloat16), batch=8)
    assert sum(rows) == 300 and rows[-1] == 4
    assert max(rows) * 2 * wide <= 256 << 20
    rows.clear()
    model.predict(torch.zeros((300, 8), dtype=torch.bfloat16), batch=150)
    assert rows == [150, 150]
