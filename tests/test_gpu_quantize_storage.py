"""GPU: the register quantizer for every storage type and mode at the edges of its tile widths, the per-tensor pair of
launches and the flat dequantizer, against the oracle's f64 arithmetic: codes, scales and zero points bit for bit."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

# one vector, below / at / above a warp's vector tiles of f32 and of the 16-bit types, whole-CTA tiles, rows that are not
# whole vectors at every width of the element kernel, rows too long for registers
COLS = [1, 8, 124, 128, 132, 256, 257, 264, 1000, 1024, 1025, 1032, 2048, 4096, 4097, 8184, 8192, 8200, 16392, 32772, 65544]


def _cfg(bits, mode, gran):
    from shrew_b200.quantize import QuantBits, QuantConfig, QuantGranularity, QuantMode
    return QuantConfig(QuantBits.Int8 if bits == 8 else QuantBits.Int4, QuantMode.Asymmetric if mode else QuantMode.Symmetric,
                       QuantGranularity.PerChannel if gran else QuantGranularity.PerTensor)


def _weights(rows, cols, mode):
    rng = np.random.default_rng(rows * 7 + cols)
    w = (rng.standard_normal((rows, cols)) * 0.3 + (0.2 if mode else 0.0)).astype(np.float32)
    flat = w.reshape(-1)
    flat[:: 97] *= 50.0
    if rows > 6:
        w[1] = 0.0                      # scale 1
        w[2, -1] = np.nan               # code 0
        w[3] = 3.0 + w[3] * 1e-4        # one-sided, narrow: a zero point far outside the codes
        w[4, 0] = np.inf                # no ordinary reciprocal
        w[5] *= 1e-32                   # below the smallest scale
    return w


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
@pytest.mark.parametrize("bits,mode", [(8, 0), (8, 1), (4, 0), (4, 1)])
@pytest.mark.parametrize("gran", [1, 0])
def test_codes_scales_and_zero_points_match_the_oracle(oracle, dtype, bits, mode, gran):
    from shrew_b200 import quantize_tensor
    for cols in COLS:
        rows = 9 if cols < 20000 else 3
        # per-tensor: the special rows would leave nothing but special values, so they go per-channel only
        w = torch.from_numpy(_weights(rows if gran else 5, cols, mode)).to(dtype)
        wide = w.float().numpy()
        qt = quantize_tensor(w.cuda(), _cfg(bits, mode, gran))
        with np.errstate(all="ignore"):
            q_ref, s_ref, z_ref = oracle.np_quantize_f32_ex(wide, gran, bits, mode)
        np.testing.assert_array_equal(qt.data.cpu().numpy().reshape(wide.shape), q_ref, err_msg=f"cols {cols}")
        np.testing.assert_array_equal(qt.scales.cpu().numpy(), s_ref)
        if mode:
            np.testing.assert_array_equal(qt.zero_points_t.cpu().numpy(), z_ref)


@pytest.mark.parametrize("gran", [1, 0])
def test_values_at_rounding_boundaries(oracle, gran):
    # every half-way point between codes and its f32 neighbours: the elements that the f32 shortcut must hand over
    from shrew_b200 import quantize_tensor
    half = (np.arange(-127, 127) + 0.5).astype(np.float32)
    row = np.concatenate([[127.0], half, np.nextafter(half, np.float32(np.inf)), np.nextafter(half, np.float32(-np.inf))]).astype(np.float32)
    w = np.stack([row * np.float32(s) for s in (1.0, 0.37, 1e-3, 7777.0, 3e-20)])
    qt = quantize_tensor(torch.from_numpy(w).cuda(), _cfg(8, 0, gran))
    q_ref, s_ref, _ = oracle.np_quantize_f32_ex(w, gran, 8, 0)
    np.testing.assert_array_equal(qt.data.cpu().numpy().reshape(w.shape), q_ref)
    np.testing.assert_array_equal(qt.scales.cpu().numpy(), s_ref)


def test_a_model_of_every_row_width_in_one_call(oracle):
    from shrew_b200 import QuantConfig
    from shrew_b200.quantize import quantize_tensors
    ws = [_weights(9, c, 0) for c in COLS]
    for gran, cfg in ((1, QuantConfig.int8_per_channel()), (0, QuantConfig.int8())):
        for w, qt in zip(ws, quantize_tensors([torch.from_numpy(w).cuda() for w in ws], cfg)):
            with np.errstate(all="ignore"):
                q_ref, s_ref, _ = oracle.np_quantize_f32_ex(w, gran, 8, 0)
            np.testing.assert_array_equal(qt.data.cpu().numpy().reshape(w.shape), q_ref, err_msg=str(w.shape))
            np.testing.assert_array_equal(qt.scales.cpu().numpy(), s_ref)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("gran", [1, 0])
def test_dequantize_in_flat_order(oracle, dtype, gran):
    # words of four codes that straddle rows (any row length), tails, rows shorter than a word
    from shrew_b200 import dequantize_tensor, quantize_tensor
    for rows, cols in ((700, 3), (701, 4), (501, 5), (333, 257), (4099, 1023), (3, 40001), (1, 1)):
        w = np.random.default_rng(cols).standard_normal((rows, cols)).astype(np.float32) * np.float32(0.02)
        qt = quantize_tensor(torch.from_numpy(w).cuda(), _cfg(8, 0, gran))
        qt.original_dtype = dtype
        q, s = qt.data.cpu().numpy().reshape(rows, cols), qt.scales.cpu().numpy()
        ref = oracle.dequantize(q, s, gran, "bf16" if dtype is torch.bfloat16 else "f32")
        back = dequantize_tensor(qt).cpu()
        back = back.view(torch.int16).numpy() if dtype is torch.bfloat16 else back.numpy()
        assert back.tobytes() == ref.tobytes(), (rows, cols)


def test_more_channels_than_a_grid_has_blocks():
    # 2^31 rows of one bf16 element: left to the kernel whose grid strides (40 GB in all)
    from shrew_b200 import quantize_tensor
    if torch.cuda.mem_get_info()[0] < 60e9:
        pytest.skip("needs 60 GB free")
    rows = 1 << 31
    w = torch.ones((rows, 1), dtype=torch.bfloat16, device="cuda")
    w[-1] = -3.0
    qt = quantize_tensor(w, _cfg(8, 0, 1))
    assert qt.scales.numel() == rows and qt.scales[0].item() == 1.0 / 127.0 and qt.scales[-1].item() == 3.0 / 127.0
    assert qt.data[-1].item() == -127 and int(qt.data[:-1].min()) == 127
    del w, qt
    torch.cuda.empty_cache()
