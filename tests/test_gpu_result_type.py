"""GPU: the sums of a forward do not depend on the type of its result.

A bf16 result is the f32 result rounded once: both are asked of the default route of one layer and compared bit for bit.
A route that sums fewer, longer chains for bf16 results only (where the rounding hides most of what that loses) fails.
"""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _layer(N, K, seed):
    from shrew_b200 import Linear, QuantConfig, QuantizedLinear
    gen = torch.Generator(device="cuda").manual_seed(seed)
    return QuantizedLinear.from_linear(Linear(torch.randn((N, K), device="cuda", generator=gen) * 0.02), QuantConfig.int8_per_channel())


def _x(M, K):
    return torch.randn((M, K), device="cuda", generator=torch.Generator(device="cuda").manual_seed(M)).to(torch.bfloat16)


# CTA pairs whose tiles are split along K (16 channel pairs, K = 11008): four ways at 200 tokens, two ways up to 512
@pytest.mark.parametrize("M,N,K", [(200, 4096, 11008), (384, 4096, 11008), (512, 4096, 11008)])
def test_bf16_result_is_the_rounded_f32_result(M, N, K):
    ql, x = _layer(N, K, N + K), _x(M, K)
    assert torch.equal(ql.forward(x), ql.forward(x, out_dtype=torch.float32).to(torch.bfloat16))
