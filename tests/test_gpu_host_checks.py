"""GPU: what the compiled host path refuses before anything is launched."""
import dataclasses

import pytest
import torch

pytestmark = pytest.mark.gpu


def _layers():
    from shrew_b200 import Linear, QuantConfig, QuantizedLinear
    return [QuantizedLinear.from_linear(Linear(torch.randn(64, 128, device="cuda")), QuantConfig.int8_per_channel()) for _ in range(2)]


def _refused(f):
    from shrew_b200 import ShrewError, _lib
    with pytest.raises(ShrewError) as e:
        f()
    assert e.value.code == _lib.ERR_INVALID_ARG


def test_output_buffers_off_the_device_or_of_another_form_are_refused():
    gate, up = _layers()
    x = torch.randn(4, 128, device="cuda")
    for bad in (torch.empty(4, 64), torch.empty(4, 64, device="cuda", dtype=torch.float16), torch.empty(4, 65, device="cuda"),
                torch.empty(3, 64, device="cuda"), torch.empty(64, 4, device="cuda").t()):
        _refused(lambda: gate.forward(x, out=bad))
        _refused(lambda: gate.forward_gate_up_silu(up, x, out=bad))
    with pytest.raises(TypeError, match="forward: out_dtype"):
        gate.forward(x, out_dtype="bf16")
    assert torch.isfinite(gate.forward(x)).all()


@pytest.mark.parametrize("gran", [0, 1])
def test_dequantize_refuses_what_does_not_cover_the_shape(gran):
    from shrew_b200 import QuantConfig, dequantize_tensor, quantize_tensor
    cfg = (QuantConfig.int8_per_channel() if gran else QuantConfig.int8()).asymmetric()
    w = torch.randn(6, 40, device="cuda")
    qt = quantize_tensor(w, cfg)
    for change in (dict(shape=[7, 40]), dict(shape=[6, 41]), dict(data=qt.data[:-1]), dict(data=qt.data.to(torch.int32)), dict(scales=qt.scales.cpu()),
                   dict(scales=qt.scales.float()), dict(scales=qt.scales[:-1]), dict(zero_points_t=qt.zero_points_t.cpu()),
                   dict(zero_points_t=qt.zero_points_t[:-1])):
        _refused(lambda: dequantize_tensor(dataclasses.replace(qt, **change)))
    with pytest.raises(TypeError, match="dequantize_tensor: the target dtype"):
        dequantize_tensor(dataclasses.replace(qt, original_dtype="f32"))
    back = dequantize_tensor(qt)
    strided = torch.empty(480, dtype=torch.int8, device="cuda")[::2]
    strided.copy_(qt.data)
    assert torch.equal(dequantize_tensor(dataclasses.replace(qt, data=strided)), back)


def test_a_gated_pair_takes_rows_of_any_rank():
    gate, up = _layers()
    x = torch.randn(5, 1, 128, device="cuda")
    ref = gate.forward_gate_up_silu(up, x[:, 0])
    assert torch.equal(gate.forward_gate_up_silu(up, x), ref)
    out = torch.empty(5, 1, 64, device="cuda")
    assert gate.forward_gate_up_silu(up, x, out=out) is out and torch.equal(out[:, 0], ref)
    _refused(lambda: gate.forward_gate_up_silu(up, torch.randn(5, 2, 128, device="cuda")))
    _refused(lambda: gate.forward(x))       # as ever: forward takes [M, in_features]
