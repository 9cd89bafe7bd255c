"""Host-side marshalling of the Python mirror that only a GPU run would otherwise exercise: the calls are
made against a recording stand-in for the library (CPU tensors carry the pointers), so a wrong field
order or a dropped tensor shows up here and not in a GPU session."""
import ctypes
import importlib.util

import pytest
import torch

from shrew_b200 import QuantConfig, QuantGranularity, _lib, build
from shrew_b200 import quantize as Q


class _FakeDevice:
    handle = ctypes.c_void_p(0x1234)

    def bind_stream(self):
        pass


class _FakeLib:
    def __init__(self):
        self.calls = []

    def shrewq_quantize_f32_batch(self, handle, items, n, gran):
        arr = ctypes.cast(items, ctypes.POINTER(_lib.QuantItem * n)).contents
        self.calls.append((gran, [(it.w_dev, it.rows, it.cols, it.q_dev, it.scales_dev) for it in arr]))
        return 0


@pytest.fixture(scope="module")
def host_ext(tmp_path_factory):
    """The compiled host path (csrc/host_path.cpp) built for CPU tensors: the same code, its allocations and device checks on the CPU
    device and no stream lookup."""
    out = str(tmp_path_factory.mktemp("host") / "_host.so")
    build.compile_host_extension(out, ["-DSHREWQ_CPU_EMU", "-O0"])
    spec = importlib.util.spec_from_file_location("_host", out)
    ext = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(ext)
    return ext


def _bind(ext, lib, error=Q.ShrewError):
    """Binds the extension to the methods of a Python stand-in: one C callback per entry point of the ABI."""
    keep = []

    def address(name):
        res, argtypes = _lib.SIGNATURES[name]
        fn = getattr(lib, name, None)
        if fn is None:
            fn = (lambda *a: 0)
        cb = ctypes.CFUNCTYPE(ctypes.c_void_p if res is ctypes.c_char_p else res, *argtypes)(fn)
        keep.append(cb)
        return ctypes.cast(cb, ctypes.c_void_p).value

    ext.bind({n: address(n) for n in _lib.SIGNATURES}, error, lambda index: _FakeDevice.handle.value)
    return keep


@pytest.fixture
def fake(monkeypatch, host_ext):
    lib = _FakeLib()
    monkeypatch.setattr(Q.Device, "get", classmethod(lambda cls, dev: _FakeDevice()))
    monkeypatch.setattr(_lib, "lib", lambda: lib)
    monkeypatch.setattr(Q, "_host", host_ext)
    lib.keep = _bind(host_ext, lib)
    return lib


def test_quantize_tensors_builds_one_table_per_granularity(fake):
    ws = [torch.zeros(6, 10), torch.zeros(3, 4, 5), torch.zeros(()), torch.zeros(0, 7), torch.zeros(1, 9)]
    out = Q.quantize_tensors(ws, QuantConfig.int8_per_channel())
    assert [t.shape for t in out] == [[6, 10], [3, 4, 5], [], [0, 7], [1, 9]]
    assert [t.scales.numel() for t in out] == [6, 3, 1, 0, 1]
    assert [t.data.numel() for t in out] == [60, 60, 1, 0, 9]
    # the rank-0 tensor goes in a per-tensor call of its own (quantize.rs:276-278), the others in one per-channel call
    assert [g for g, _ in fake.calls] == [QuantGranularity.PerChannel.value, QuantGranularity.PerTensor.value]
    main, single = fake.calls[0][1], fake.calls[1][1]
    assert [(r, c) for _, r, c, _, _ in main] == [(6, 10), (3, 20), (0, 7), (1, 9)]
    assert [(r, c) for _, r, c, _, _ in single] == [(1, 1)]
    for (w_ptr, _, _, q_ptr, s_ptr), w, t in zip(main, [ws[0], ws[1], ws[3], ws[4]], [out[0], out[1], out[3], out[4]]):
        assert w_ptr == (w.data_ptr() or None) and q_ptr == (t.data.data_ptr() or None) and s_ptr == (t.scales.data_ptr() or None)
    assert single[0][0] == ws[2].data_ptr() and single[0][3] == out[2].data.data_ptr()


def test_quantize_tensors_per_tensor_config_is_one_call(fake):
    out = Q.quantize_tensors([torch.zeros(4, 4), torch.zeros(())], QuantConfig.int8())
    assert len(fake.calls) == 1 and fake.calls[0][0] == QuantGranularity.PerTensor.value
    assert [t.scales.numel() for t in out] == [1, 1]


def test_quantize_tensors_refuses_what_the_kernels_do_not_take(fake):
    with pytest.raises(Q.ShrewError):
        Q.quantize_tensors([torch.zeros(2, 2, dtype=torch.bfloat16)], QuantConfig.int8())
    with pytest.raises(Q.ShrewError):
        Q.quantize_tensors([torch.zeros(2, 2)], QuantConfig.int4())
    assert Q.quantize_tensors([], QuantConfig.int8()) == [] and fake.calls == []


def test_named_parameters_walk_goes_out_as_one_batch(fake):
    class M:
        def named_parameters(self):
            return [("weight", torch.zeros(4, 8)), ("bias", torch.zeros(1, 4)), ("gain", torch.zeros(4))]

    out = Q.quantize_named_parameters(M(), QuantConfig.int8())
    assert [n for n, _ in out] == ["weight", "bias"]            # rank >= 2 only, the [1, out] bias included (quantize.rs:507-513)
    assert len(fake.calls) == 1 and len(fake.calls[0][1]) == 2


class _SignatureCheckingLib:
    """Stands in for libshrewq: every call must carry as many arguments as the C declaration has parameters,
    each acceptable to its ctypes type; returns success."""

    def __init__(self):
        self.calls = []

    def __getattr__(self, name):
        if name not in _lib.SIGNATURES:
            raise AttributeError(name)
        res, argtypes = _lib.SIGNATURES[name]

        def call(*args):
            assert len(args) == len(argtypes), f"{name}: {len(args)} arguments for {len(argtypes)} parameters"
            for a, t in zip(args, argtypes):
                t.from_param(a)
            self.calls.append(name)
            return None if res is ctypes.c_char_p else 0
        return call


def test_every_mode_of_the_python_mirror_marshals_its_call(monkeypatch, host_ext):
    # the experimental modes (asymmetric, INT4, other storage types, packed INT4, shard entry points) have not
    # run on a GPU; their host side at least calls the C ABI with the declared arity and types
    from shrew_b200 import Linear, quantization_stats, quantize_named_parameters
    lib = _SignatureCheckingLib()
    monkeypatch.setattr(Q.Device, "get", classmethod(lambda cls, dev: _FakeDevice()))
    monkeypatch.setattr(_lib, "lib", lambda: lib)
    monkeypatch.setattr(Q, "_host", host_ext)
    keep = _bind(host_ext, lib)
    w = torch.randn(8, 128)
    for cfg in (QuantConfig.int8(), QuantConfig.int8_per_channel(), QuantConfig.int4_per_channel(), QuantConfig.int8().asymmetric()):
        for dt in (torch.float32, torch.bfloat16, torch.float16, torch.float64):
            qt = Q.quantize_tensor(w.to(dt), cfg)
            for back in (Q.dequantize_tensor(qt), Q.dequantize_tensor(qt, device="cuda")):
                assert list(back.shape) == [8, 128] and back.dtype == dt
            assert (qt.zero_points_t is not None) == (cfg.mode is Q.QuantMode.Asymmetric)
    shard = Q.quantize_tensor_given_amax(w, Q.absmax(w))
    assert shard.scales.numel() == 1
    Q.QuantizedLinear.new(Q.quantize_tensor(w, QuantConfig.int8_per_channel()), torch.zeros(8))
    Q.QuantizedLinear.new(Q.quantize_tensor(w, QuantConfig.int8_per_channel().asymmetric()), None)
    q4 = Q.quantize_tensor(w, QuantConfig.int4_per_channel())
    assert Q.pack_int4(q4).numel() == 8 * 128 // 2
    Q.QuantizedLinear.new_int4_packed(q4, None)
    lin = Linear(w, torch.zeros(8))
    assert len(quantize_named_parameters(lin, QuantConfig.int8())) == 2
    assert quantization_stats(lin, QuantConfig.int8()).num_quantized == 2
    assert {"shrewq_quantize_f32", "shrewq_quantize_f32_ex", "shrewq_quantize_any", "shrewq_dequantize", "shrewq_dequantize_ex",
            "shrewq_absmax_f32", "shrewq_quantize_f32_given_amax", "shrewq_linear_create", "shrewq_linear_create_ex",
            "shrewq_pack_int4", "shrewq_linear_create_int4"} <= set(lib.calls)
    del keep


def test_without_a_device_every_entry_raises():
    for f in (lambda t: Q.quantize_tensor(t, QuantConfig.int8()), lambda t: Q.quantize_tensors([t], QuantConfig.int8()), Q.absmax,
              lambda t: Q.dequantize_tensor(Q.QuantizedTensor(t.to(torch.int8), t.double(), [4], torch.float32))):
        with pytest.raises(Q.ShrewError) as e:
            f(torch.zeros(4))
        assert e.value.code == _lib.ERR_NO_DEVICE


# ---- the compiled forward ---------------------------------------------------------------------------------
class _ForwardLib:
    def __init__(self, rc=0):
        self.calls, self.rc = [], rc
        self.message = ctypes.create_string_buffer(b"from the library")

    def shrewq_linear_forward(self, *a):
        self.calls.append(a)
        return self.rc

    def shrewq_linear_forward_gate_up_silu(self, *a):
        self.calls.append(a)
        return self.rc

    def shrewq_last_error(self, ctx):
        return ctypes.addressof(self.message)


def test_compiled_forward_marshals_its_call(host_ext):
    lib = _ForwardLib()
    keep = _bind(host_ext, lib)
    layer, up = host_ext.Layer(0x1234, 0x77, 0, 8, 3), host_ext.Layer(0x1234, 0x78, 0, 8, 3)
    x = torch.zeros(5, 16)[:, ::2]                                   # strided: copied
    y = layer.forward(x, 1, None, torch.bfloat16)
    assert y.shape == (5, 3) and y.dtype is torch.bfloat16
    (h, xp, xt, M, yp, yt, ldy, epilogue), = lib.calls
    assert (h, xt, M, yp, yt, ldy, epilogue) == (0x77, _lib.F32, 5, y.data_ptr(), _lib.BF16, 3, 1) and xp not in (None, x.data_ptr())
    wide = torch.zeros(5, 10)
    x = torch.zeros(5, 8, dtype=torch.bfloat16)
    assert layer.forward(x, 0, wide[:, 4:7], None).data_ptr() == wide[:, 4:7].data_ptr()
    assert lib.calls[-1] == (0x77, x.data_ptr(), _lib.BF16, 5, wide.data_ptr() + 16, _lib.F32, 10, 0)
    h = layer.gate_up_silu(up, x.view(5, 1, 8), None)
    assert lib.calls[-1] == (0x77, 0x78, x.data_ptr(), _lib.BF16, 5, h.data_ptr(), _lib.BF16, 3)
    del keep


def test_compiled_forward_refuses_before_the_call(host_ext):
    lib = _ForwardLib()
    keep = _bind(host_ext, lib)
    layer = host_ext.Layer(0x1234, 0x77, 0, 8, 3)
    x = torch.zeros(5, 8)
    for args, code in (((torch.zeros(5, 7), 0, None, None), _lib.ERR_INVALID_ARG), ((x.double(), 0, None, None), _lib.ERR_UNSUPPORTED),
                       ((x, 0, None, torch.float16), _lib.ERR_UNSUPPORTED), ((x, 0, torch.zeros(4, 3), None), _lib.ERR_INVALID_ARG),
                       ((x, 0, torch.zeros(3, 5).t(), None), _lib.ERR_INVALID_ARG), ((x, 0, torch.zeros(5, 3, device="meta"), None), _lib.ERR_INVALID_ARG),
                       ((x.to("meta"), 0, None, None), _lib.ERR_INVALID_ARG)):
        with pytest.raises(Q.ShrewError) as e:
            layer.forward(*args)
        assert e.value.code == code
    for bad in ((x, 0, None), (x, "relu", None, None), ([1.0], 0, None, None), (x, 0, None, "bf16")):
        with pytest.raises(TypeError):
            layer.forward(*bad)
    with pytest.raises(TypeError):
        layer.gate_up_silu(None, x, None)
    assert lib.calls == []
    lib.rc = _lib.ERR_CUDA
    with pytest.raises(Q.ShrewError, match="from the library") as e:
        layer.forward(x, 0, None, None)
    assert e.value.code == _lib.ERR_CUDA
    del keep


def test_compiled_dequantize_refuses_before_the_call(host_ext):
    class Lib:
        calls = 0

        def shrewq_dequantize_ex(self, *a):
            Lib.calls += 1
            return 0

    keep = _bind(host_ext, Lib())
    q, s = torch.zeros(12, dtype=torch.int8), torch.ones(3, dtype=torch.float64)
    for args in ((q, s, None, [4, 4], False), (q.int(), s, None, [3, 4], True), (q, s.float(), None, [3, 4], True), (q, s[:2], None, [3, 4], True),
                 (q, s, s[:2], [3, 4], True), (q, s.to("meta"), None, [3, 4], True)):
        with pytest.raises(Q.ShrewError) as e:
            host_ext.dequantize(*args, torch.float32)
        assert e.value.code == _lib.ERR_INVALID_ARG
    assert Lib.calls == 0
    assert host_ext.dequantize(q, s, None, [3, 4], True, torch.float32).shape == (3, 4) and Lib.calls == 1
    del keep


def test_quantized_linear_module_surface_without_a_device():
    # the Module methods a QuantizedLinear inherits (quantize.rs:462-482 overrides only forward and parameters):
    # pure host state, checked on an instance that never touched the library
    ql = object.__new__(Q.QuantizedLinear)
    ql._h = None
    assert ql.parameters() == [] and ql.named_parameters() == []
    assert ql.num_parameters() == 0 and ql.trainable_params_count() == 0
    assert ql.is_training() is True
    ql.set_training(False)
    assert ql.is_training() is False


def test_forward_host_marshals_host_pointers_and_checks_its_input(monkeypatch):
    calls = []

    class Lib:
        def shrewq_linear_forward_host(self, h, x, x_dtype, M, y, y_dtype, epilogue):
            calls.append((h, x.value, x_dtype, M, y.value, y_dtype, epilogue))
            return 0

    monkeypatch.setattr(_lib, "lib", lambda: Lib())
    ql = object.__new__(Q.QuantizedLinear)
    ql._h, ql.in_features, ql.out_features, ql.device = 0x77, 8, 3, _FakeDevice()
    x = torch.zeros(5, 8, dtype=torch.bfloat16)
    y = ql.forward_host(x, epilogue=1, out_dtype=torch.float32)
    assert y.shape == (5, 3) and y.dtype == torch.float32 and y.device.type == "cpu"
    (h, xp, xd, M, yp, yd, ep), = calls
    assert (h, xp, xd, M, yp, yd, ep) == (0x77, x.data_ptr(), _lib.BF16, 5, y.data_ptr(), _lib.F32, 1)
    with pytest.raises(Q.ShrewError):
        ql.forward_host(torch.zeros(5, 7))                       # wrong in_features
    with pytest.raises(Q.ShrewError):
        ql.forward_host(torch.zeros(5, 8, dtype=torch.float64))  # unsupported dtype
    ql._h = None
