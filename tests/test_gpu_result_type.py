"""GPU: the sums of a forward do not depend on the type of its result.

A bf16 result is the f32 result rounded once: both are asked of the default route of one layer and compared bit for bit.
A route that sums fewer, longer chains for bf16 results only (where the rounding hides most of what that loses) fails.
"""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _layer(N, K, seed, bias=False):
    from shrew_b200 import Linear, QuantConfig, QuantizedLinear
    gen = torch.Generator(device="cuda").manual_seed(seed)
    w = torch.randn((N, K), device="cuda", generator=gen) * 0.02
    b = torch.randn(N, device="cuda", generator=gen) if bias else None
    return QuantizedLinear.from_linear(Linear(w, b), QuantConfig.int8_per_channel())


def _x(M, K):
    return torch.randn((M, K), device="cuda", generator=torch.Generator(device="cuda").manual_seed(M)).to(torch.bfloat16)


# CTA pairs whose tiles are split along K (16 channel pairs, K = 11008): four ways at 200 tokens, two ways up to 512; 17 to 32 and two
# tokens on weights from 2^25 codes on
@pytest.mark.parametrize("M,N,K", [(200, 4096, 11008), (384, 4096, 11008), (512, 4096, 11008), (17, 11008, 4096), (32, 4096, 11008),
                                   (2, 11008, 4096), (2, 4096, 11008)])
def test_bf16_result_is_the_rounded_f32_result(M, N, K):
    ql, x = _layer(N, K, N + K), _x(M, K)
    assert torch.equal(ql.forward(x), ql.forward(x, out_dtype=torch.float32).to(torch.bfloat16))


def _run(kind, f):
    from shrew_b200 import _lib
    _lib.lib().shrewq_force_kernel(kind.encode())
    try:
        return f()
    finally:
        _lib.lib().shrewq_force_kernel(b"auto")


# 17 to 32 tokens: the default route gives the register-streaming kernel's results bit for bit, on both sides of the token blocks
# of 8, of a stage of 2048 features and of one row block per CTA, with and without bias
@pytest.mark.parametrize("M,N,K,bias", [(17, 4096, 4096, True), (24, 4096, 4096, False), (25, 11008, 4096, True), (32, 4096, 11008, True),
                                        (32, 40, 2112, True), (19, 7, 64, True), (24, 20000, 2048, True)])
def test_17_to_32_tokens_are_summed_as_by_the_register_streaming_kernel(M, N, K, bias):
    ql, x = _layer(N, K, N + K, bias), _x(M, K)
    for out_dtype in (torch.float32, torch.bfloat16):
        y = ql.forward(x, out_dtype=out_dtype)
        assert ql.last_kernel() == "mma-ring"
        assert torch.equal(y, _run("mma", lambda: ql.forward(x, out_dtype=out_dtype)))


@pytest.mark.parametrize("M,N,K", [(17, 11008, 4096), (24, 520, 2048), (27, 11008, 4096), (32, 1030, 4160)])
def test_17_to_32_tokens_of_a_gated_pair(M, N, K):
    gate, up, x = _layer(N, K, 1, True), _layer(N, K, 2, True), _x(M, K)
    for dtype in (torch.float32, torch.bfloat16):
        out = [torch.empty((M, N), dtype=dtype, device="cuda") for _ in range(2)]
        gate.forward_gate_up_silu(up, x, out=out[0])
        assert gate.last_kernel() == "mma-ring"
        _run("mma", lambda: gate.forward_gate_up_silu(up, x, out=out[1]))
        assert torch.equal(*out)


# Up to 16 tokens the same holds from more than five CTAs of 16 rows per SM on
@pytest.mark.parametrize("M,rows_per_sm,gated", [(3, 81, False), (8, 200, False), (16, 81, False), (9, 41, True), (16, 75, True)])
def test_large_grids_are_summed_as_by_the_register_streaming_kernel(M, rows_per_sm, gated):
    N = rows_per_sm * torch.cuda.get_device_properties(0).multi_processor_count
    gate, x = _layer(N, 2176, 5, True), _x(M, 2176)
    up = _layer(N, 2176, 6) if gated else None
    for dtype in (torch.float32, torch.bfloat16):
        out = [torch.empty((M, N), dtype=dtype, device="cuda") for _ in range(2)]
        for y, kind in zip(out, ("auto", "mma")):
            _run(kind, lambda: gate.forward_gate_up_silu(up, x, out=y) if gated else gate.forward(x, out=y))
            assert gate.last_kernel() == ("mma" if kind == "mma" else "mma-ring")
        assert torch.equal(*out)


# These calls need no workspace of the context: the first one of a new context can be captured, and calls on two streams share
# nothing.
@pytest.mark.parametrize("M", [24, 64])
def test_a_gated_pair_with_a_short_last_wave_captures_without_a_warm_up(M, monkeypatch):
    from shrew_b200 import QuantizedLinear
    from shrew_b200.quantize import Device
    weights = [_layer(11008, 4096, seed).weight_q for seed in (3, 4)]
    monkeypatch.setitem(Device._by_index, torch.cuda.current_device(), Device(torch.cuda.current_device()))
    (gate, up), x = [QuantizedLinear(w, None) for w in weights], _x(M, 4096)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        y = gate.forward_gate_up_silu(up, x)
    g.replay()
    assert torch.equal(y, gate.forward_gate_up_silu(up, x))
