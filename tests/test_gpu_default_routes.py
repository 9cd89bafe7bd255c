"""GPU: the default route (no kernel forced) against the oracle at sizes on both sides of each rule of the dispatch."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

TOL_F32, TOL_BF16 = 1e-4, 1e-2     # the forward's stated tolerances by activation type


@pytest.fixture(autouse=True)
def _options():
    yield
    from shrew_b200.quantize import Device
    for name, value in (("tc_f32", 1), ("pdl", 1)):
        Device.get("cuda").set_option(name, value)


def _layer(N, K, seed, bias=True):
    from shrew_b200 import Linear, QuantConfig, QuantizedLinear
    rng = np.random.default_rng(seed)
    w = (rng.standard_normal((N, K)) * 0.05).astype(np.float32)
    b = (rng.standard_normal(N) * 0.1).astype(np.float32) if bias else None
    return QuantizedLinear.from_linear(Linear(torch.from_numpy(w).cuda(), None if b is None else torch.from_numpy(b).cuda()),
                                       QuantConfig.int8_per_channel())


def _ref(oracle, ql, x, relu=False):
    q = ql.weight_q.data.cpu().numpy().reshape(ql.out_features, ql.in_features)
    b = None if ql.bias is None else ql.bias.cpu().numpy().reshape(-1)
    return oracle.np_linear_forward(q, ql.weight_q.scales.cpu().numpy(), 1, b, x, relu=relu)


def _launches(f):
    from shrew_b200.quantize import Device
    dev = Device.get("cuda")
    before = dev.launch_count()
    y = f()
    return y, dev.launch_count() - before


# f32 activations.  Persistent kernel (one launch) up to 1024 features and f32 results: activations resident or not (512 and 768
# features at 64 tokens a tile, 256 and 384 at 128), one and several tiles per CTA, output rows off a sector.  The split copy and the
# pipeline over it (two launches) beyond, and for bf16 results.
@pytest.mark.parametrize("M,N,K,out,launches", [
    (300, 130, 512, "f32", 1), (200, 200, 528, "f32", 1), (250, 333, 784, "f32", 1), (300, 129, 1024, "f32", 1),
    (2100, 1304, 256, "f32", 1), (2100, 1303, 256, "f32", 1), (1300, 2001, 400, "f32", 1), (1300, 2008, 1024, "f32", 1),
    (300, 130, 1040, "f32", 2), (520, 700, 2048, "f32", 2), (200, 256, 4096, "f32", 2), (300, 130, 512, "bf16", 2), (520, 1000, 2048, "bf16", 2)])
def test_f32_activations(oracle, M, N, K, out, launches):
    ql = _layer(N, K, M + N)
    x = np.random.default_rng(K).random((M, K), dtype=np.float32)
    dtype = torch.float32 if out == "f32" else torch.bfloat16
    xd = torch.from_numpy(x).cuda()
    ql.forward(xd, out_dtype=dtype)     # (workspaces)
    y, n = _launches(lambda: ql.forward(xd, epilogue=1, out_dtype=dtype))
    assert ql.last_kernel() == "tcgen05-f32" and n == launches
    assert oracle.rel_err(y.float().cpu().numpy(), _ref(oracle, ql, x, relu=True)) < (TOL_F32 if out == "f32" else TOL_BF16)


# the persistent kernel and the pipeline on the same call, on each side of 1024 features: both split x into bf16 hi + lo (2^-17 of each
# value) and sum in f32, so they agree to a few times that
@pytest.mark.parametrize("M,N,K", [(300, 700, 1024), (300, 700, 1040), (1300, 1000, 2048)])
def test_both_f32_kernels_agree(oracle, M, N, K):
    from shrew_b200.quantize import Device
    ql = _layer(N, K, K)
    x = torch.rand((M, K), device="cuda")
    y = []
    for option, launches in ((0, 2), (2, 1)):
        Device.get("cuda").set_option("tc_f32", option)
        ql.forward(x)
        out, n = _launches(lambda: ql.forward(x))
        assert n == launches
        y.append(out.cpu().numpy())
    ref = _ref(oracle, ql, x.cpu().numpy())
    assert all(oracle.rel_err(v, ref) < TOL_F32 for v in y) and oracle.rel_err(y[0], y[1]) < 2e-5


# bf16 activations: both result types, ragged sizes, at the edges of the families' batch ranges and of their tiles
@pytest.mark.parametrize("M,N,K,kernel", [
    (1, 1000, 4096, "gemv"), (2, 11008, 4096, "gemv"), (3, 1000, 4160, "mma-ring"), (16, 24000, 512, "mma-ring"), (17, 11008, 4096, "mma-ring"),
    (32, 1001, 4160, "mma-ring"), (33, 20000, 1024, "tcgen05"), (64, 24000, 512, "tcgen05"), (128, 1000, 2064, "tcgen05"),
    (200, 4096, 11008, "tcgen05-2cta"), (300, 4100, 8208, "tcgen05-2cta"), (500, 11008, 1040, "tcgen05-2cta")])
def test_bf16_activations(oracle, M, N, K, kernel):
    ql = _layer(N, K, M + K)
    x = torch.from_numpy(np.random.default_rng(M).random((M, K), dtype=np.float32)).cuda().to(torch.bfloat16)
    ref = _ref(oracle, ql, x.float().cpu().numpy())
    for dtype, tol in ((torch.bfloat16, TOL_BF16), (torch.float32, 1e-5)):   # exact products, f32 sums: K * 2^-24 at most
        y = ql.forward(x, out_dtype=dtype)
        assert ql.last_kernel() == kernel
        assert oracle.rel_err(y.float().cpu().numpy(), ref) < tol


# gated pairs: f32 slices of 4 tokens, the ring kernel on both sides of 16 tokens, a short last wave of small tiles, ragged pairs
@pytest.mark.parametrize("M,N,K,x", [(20, 70, 512, "f32"), (33, 33, 1040, "f32"), (17, 11008, 4096, "bf16"), (32, 6001, 2112, "bf16"),
                                     (64, 11008, 1024, "bf16"), (300, 8200, 528, "bf16")])
def test_gated_pairs(oracle, M, N, K, x):
    gate, up = _layer(N, K, 1), _layer(N, K, 2)
    xd = torch.from_numpy(np.random.default_rng(M).random((M, K), dtype=np.float32) - 0.3).cuda().to(torch.float32 if x == "f32" else torch.bfloat16)
    g, u = (_ref(oracle, l, xd.float().cpu().numpy()).astype(np.float64) for l in (gate, up))
    y = gate.forward_gate_up_silu(up, xd)
    assert oracle.rel_err(y.float().cpu().numpy(), g / (1 + np.exp(-g)) * u) < (TOL_F32 if x == "f32" else TOL_BF16)


# chains of layers under dependent launch: every kernel starts while the one that makes its activations still runs
@pytest.mark.parametrize("M,widths", [(300, (784, 256, 1024, 528, 256)), (64, (784, 256, 1024, 400, 16)), (40, (256, 4096, 512, 2048, 64))])
def test_chains_of_f32_layers_give_the_same_with_and_without_dependent_launch(M, widths):
    from shrew_b200.quantize import Device
    ls = [_layer(n, k, n + k) for k, n in zip(widths, widths[1:])]
    x = torch.rand((M, widths[0]), device="cuda")
    out = []
    for pdl in (0, 1):
        Device.get("cuda").set_option("pdl", pdl)
        for _ in range(20):
            y = x
            for l in ls:
                y = l.forward(y, epilogue=1)
            out.append(y)
    assert all(torch.equal(y, out[0]) for y in out)
