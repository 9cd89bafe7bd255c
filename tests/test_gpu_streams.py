"""GPU: calls on two streams of one context."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _layer(N, K):
    from shrew_b200 import Linear, QuantConfig, QuantizedLinear
    w = torch.randn((N, K), device="cuda", generator=torch.Generator(device="cuda").manual_seed(N)) * 0.02
    return QuantizedLinear.from_linear(Linear(w), QuantConfig.int8_per_channel())


def test_per_tensor_quantize_beside_a_forward_split_along_k():
    # the forward's partial sums (64 tokens, 32 channel tiles split four ways) and the quantizer's words are apart
    from shrew_b200 import QuantConfig, quantize_tensor
    ql = _layer(4096, 4096)
    x = torch.randn((64, 4096), device="cuda").to(torch.bfloat16)
    ws = [torch.randn(n, device="cuda") * s for n, s in ((1 << 20, 1.0), (3 << 20, 7.0), (1 << 22, 0.1))]
    y_ref, q_ref = ql.forward(x), [quantize_tensor(w, QuantConfig.int8()) for w in ws]
    torch.cuda.synchronize()
    side = torch.cuda.Stream()
    ys, qs = [], []
    for _ in range(40):
        ys += [ql.forward(x) for _ in range(3)]
        with torch.cuda.stream(side):
            qs.append([quantize_tensor(w, QuantConfig.int8()) for w in ws])
    torch.cuda.synchronize()
    assert all(torch.equal(y, y_ref) for y in ys)
    for q in qs:
        for a, b in zip(q, q_ref):
            assert torch.equal(a.data, b.data) and torch.equal(a.scales, b.scales)


def test_per_tensor_quantize_on_two_streams_at_once():
    from shrew_b200 import QuantConfig, quantize_tensor
    ws = [torch.randn(n, device="cuda") * s for n, s in ((5000, 1.0), (3 << 20, 7.0))]
    ref = [quantize_tensor(w, QuantConfig.int8()) for w in ws]
    streams = [torch.cuda.Stream() for _ in ws]
    torch.cuda.synchronize()
    out = []
    for _ in range(4):                   # eight calls: as many as the context keeps apart
        for s, w in zip(streams, ws):
            with torch.cuda.stream(s):
                out.append(quantize_tensor(w, QuantConfig.int8()))
    torch.cuda.synchronize()
    for i, q in enumerate(out):
        assert torch.equal(q.data, ref[i % 2].data) and torch.equal(q.scales, ref[i % 2].scales)


def test_a_per_tensor_quantize_needs_no_workspace_under_capture():
    from shrew_b200 import QuantConfig, quantize_tensor
    from shrew_b200.quantize import Device
    from shrew_b200 import _lib
    w = torch.randn(100000, device="cuda")
    ref = quantize_tensor(w, QuantConfig.int8())
    dev = Device(torch.cuda.current_device())    # a context without any workspace yet
    q, s = torch.empty_like(ref.data), torch.empty_like(ref.scales)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        dev.bind_stream()
        _lib.check(_lib.lib().shrewq_quantize_f32(dev.handle, w.data_ptr(), 1, w.numel(), _lib.PER_TENSOR, q.data_ptr(), s.data_ptr()), dev.handle)
    g.replay()
    torch.cuda.synchronize()
    assert torch.equal(q, ref.data) and torch.equal(s, ref.scales)


@pytest.mark.parametrize("gran", [0, 1])
def test_quantizers_under_both_settings_of_dependent_launch(gran):
    # back to back, each call reading what the one before wrote
    from shrew_b200 import QuantConfig, dequantize_tensor, quantize_tensor
    from shrew_b200.quantize import Device, quantize_tensors
    cfg = QuantConfig.int8_per_channel() if gran else QuantConfig.int8()
    w = torch.randn((700, 1023), device="cuda")
    dev, out = Device.get("cuda"), []
    try:
        for pdl in (0, 1):
            dev.set_option("pdl", pdl)
            qt = quantize_tensor(w, cfg)
            for _ in range(5):
                qt = quantize_tensor(dequantize_tensor(qt), cfg)
            out.append(quantize_tensors([dequantize_tensor(qt)] * 2, cfg)[1])
    finally:
        dev.set_option("pdl", 1)
    assert torch.equal(out[0].data, out[1].data) and torch.equal(out[0].scales, out[1].scales)
