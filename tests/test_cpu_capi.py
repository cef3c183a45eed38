"""The C-ABI library loads without a GPU, exports every symbol the header declares, and validates
its arguments before touching the device."""
import ctypes
import re
from pathlib import Path

import pytest

from zenith_b200 import _capi

ROOT = Path(__file__).resolve().parent.parent
HEADER = (ROOT / "include" / "zenith_b200.h").read_text()


def declared_functions():
    body = re.sub(r"/\*.*?\*/", "", HEADER, flags=re.S)
    return sorted(set(re.findall(r"\b(zen_[a-z0-9_]+)\s*\(", body)))


def test_every_declared_symbol_is_exported_and_bound():
    lib = _capi.lib()
    names = declared_functions()
    assert len(names) >= 25
    for n in names:
        assert hasattr(lib, n), f"{n} declared in include/zenith_b200.h but not exported"
        assert n in _capi.SIGNATURES, f"{n} has no ctypes prototype"
    assert set(_capi.SIGNATURES) <= set(names)


def test_version_and_status_strings():
    assert _capi.lib().zen_version() == 100
    assert _capi.status_string(0) == "ok"
    for s in range(1, 7):
        assert _capi.status_string(s) not in ("ok", "unknown status")
    assert _capi.status_string(99) == "unknown status"


def test_argument_validation_needs_no_device():
    lib = _capi.lib()
    z = None
    assert lib.zen_linear_i8(z, 16, z, 16, 1, 1, 16, 1.0, z, z, 0, 0, 1.0, 0, z, 1, z) == _capi.ERR_INVALID_ARG
    one = ctypes.c_void_p(16)  # never dereferenced: rejected before any launch
    assert lib.zen_linear_i8(one, 24, one, 24, 4, 4, 24, 1.0, z, z, 0, 0, 1.0, 0, one, 4, z) == _capi.ERR_UNSUPPORTED
    assert lib.zen_linear_i8(one, 16, one, 16, 4, 4, 16, 1.0, z, z, 9, 0, 1.0, 0, one, 4, z) == _capi.ERR_INVALID_ARG
    assert lib.zen_linear_i8(one, 16, one, 16, 4, 4, 16, 1.0, z, z, 0, 3, 0.0, 0, one, 4, z) == _capi.ERR_INVALID_ARG
    assert lib.zen_linear_f16(one, 12, one, 12, 4, 4, 12, z, 0, 2, one, 4, z) == _capi.ERR_UNSUPPORTED
    assert lib.zen_wmma_matmul_f16(one, one, one, 16, 12, 16, z) == _capi.ERR_UNSUPPORTED
    assert lib.zen_flash_attention_f16(one, one, one, one, z, 1.0, 1, 1, 8, 32, *([8] * 12), z, 0, 1.0, z) == _capi.ERR_UNSUPPORTED
    assert lib.zen_quantize_f32(one, one, 4, 0.0, 0, 0, z) == _capi.ERR_INVALID_ARG
    assert lib.zen_layernorm_f32(z, z, z, z, 4, 8, 1e-5, z) == _capi.ERR_INVALID_ARG
    # per-call options: an unknown flag bit or tile width is rejected
    ex = lambda flags: lib.zen_linear_i8_ex(one, 16, one, 16, 4, 4, 16, 1.0, z, z, 0, 0, 1.0, 0, one, 4, z, 0, z, 0, flags, z)
    assert ex(0x80) == _capi.ERR_INVALID_ARG and ex(_capi.gemm_tile_n(100)) == _capi.ERR_INVALID_ARG
    assert ex(_capi.GEMM_PAIR | _capi.GEMM_NO_PAIR) == _capi.ERR_INVALID_ARG
    attn = lambda flags: lib.zen_flash_attention_f16_ex(one, one, one, one, z, 1.0, 1, 1, 8, 32, *([8] * 12), z, 0, 1.0, flags, z)
    assert attn(_capi.ATTN_KEYS_64 | _capi.ATTN_KEYS_128) == attn(0x4) == _capi.ERR_INVALID_ARG
    assert attn(_capi.ATTN_KEYS_64) == attn(_capi.ATTN_KEYS_128) == _capi.ERR_UNSUPPORTED  # (the head size)
    # zero-sized work is a no-op, not an error
    assert lib.zen_gelu_f32(z, z, 0, z) == 0 and lib.zen_layernorm_f16(z, z, z, z, 0, 8, 1e-5, z) == 0


def test_one_launch_forms_name_what_they_do_not_take():
    """A valid call that needs the form with a workspace has a status of its own, whether size or alignment is the reason, and
    one that no form takes is refused as by the other form."""
    lib, z, one, odd = _capi.lib(), None, ctypes.c_void_p(16), ctypes.c_void_p(20)  # never dereferenced: nothing is launched
    needs = _capi.ERR_NEEDS_WORKSPACE
    assert lib.zen_matmul_f32_direct(one, one, one, 4096, 4096, 64, z) == needs
    assert lib.zen_matmul_f32_direct(one, one, one, 4096, 4096, 63, z) == _capi.ERR_UNSUPPORTED
    attn = lambda q, k, o, S, D: lib.zen_flash_attention_f32_direct(q, k, one, o, 4, 64, S, D, z, 0, 1.0, z)
    assert attn(one, one, one, 4096, 64) == attn(odd, one, one, 100, 64) == attn(one, odd, one, 100, 128) == needs
    assert attn(one, one, odd, 100, 64) == attn(one, one, one, 100, 32) == _capi.ERR_UNSUPPORTED
    assert "workspace" in _capi.status_string(needs) and _capi.status_string(needs) != _capi.status_string(_capi.ERR_TOO_LARGE)


def test_operators_refuse_cpu_tensors():
    import torch

    from zenith_b200 import zenith_cuda

    x = torch.zeros(4, 8)
    for call in (lambda: zenith_cuda.gelu(x), lambda: zenith_cuda.relu(x), lambda: zenith_cuda.layernorm(x, x[0], x[0]),
                 lambda: zenith_cuda.matmul(x, x.T), lambda: zenith_cuda.wmma_matmul(x.half(), x.T.half()),
                 lambda: zenith_cuda.flash_attention(x[None, None], x[None, None], x[None, None])):
        with pytest.raises(RuntimeError):
            call()


def test_operators_refuse_vectors_that_a_kernel_would_read_past(monkeypatch):
    """Scales, biases, LayerNorm parameters, key lengths and packed positions that are too short or on another device raise
    before anything is launched (fake CUDA tensors: no device is needed)."""
    import torch
    from torch._subclasses.fake_tensor import FakeTensorMode

    from zenith_b200 import ops

    def launched(*a):
        raise AssertionError("launched")

    monkeypatch.setattr(ops, "_call", launched)
    monkeypatch.setattr(ops, "_layernorm_workspace", lambda *a: (None, 0))
    i8, u8, i32, f16, f32 = torch.int8, torch.uint8, torch.int32, torch.float16, torch.float32
    with FakeTensorMode():
        T = lambda *shape, dt=f32, dev="cuda:0": torch.empty(shape, dtype=dt, device=dev)
        M, K, N = 4, 64, 768
        q = T(3, 2, 16, 64, dt=f16)
        x8, w8, res, h = T(M, K, dt=i8), T(N, K, dt=i8), T(M, N, dt=f16), T(N, dt=f16)
        ids, word, pos, typ = T(32, dt=i32), T(100, N, dt=f16), T(16, N, dt=f16), T(2, N, dt=f16)
        calls = {
            "kv_lens": [
                lambda n, dev="cuda:0": ops.flash_attention(q, q, q, kv_lens=T(n, dt=i32, dev=dev)),
                lambda n, dev="cuda:0": ops.flash_attention(q.float(), q.float(), q.float(), kv_lens=T(n, dt=i32, dev=dev)),
                lambda n, dev="cuda:0": ops.flash_attention_strided(q, q, q, q, 3, 2, 16, 64, *[(1, 1, 1)] * 4, kv_lens=T(n, dt=i32, dev=dev)),
                lambda n, dev="cuda:0": ops.qkv_attention_int8(T(48, K, dt=i8), T(384, K, dt=i8), 1.0, None, None, 3, 16, 2, kv_lens=T(n, dt=i32, dev=dev)),
                lambda n, dev="cuda:0": ops.pack_tokens(T(3, 16, dt=i32), T(n, dt=i32, dev=dev), 48)],
            "w_scale": [
                lambda n, dev="cuda:0": ops.linear_int8_add_layernorm(x8, w8, 1.0, T(n, dev=dev), None, res, h, h, 1e-5),
                lambda n, dev="cuda:0": ops.qkv_attention_int8(T(48, K, dt=i8), T(384, K, dt=i8), 1.0, T(n, dev=dev), None, 3, 16, 2),
                lambda n, dev="cuda:0": ops.qkv_attention_unpadded_int8(T(48, K, dt=i8), T(384, K, dt=i8), 1.0, T(n, dev=dev), None, T(4, dt=i32), 2),
                lambda n, dev="cuda:0": ops.linear_fp8(x8.view(u8), w8.view(u8), 1.0, T(n, dev=dev))],
            "bias": [
                lambda n, dev="cuda:0": ops.linear_fp16(T(M, K, dt=f16), T(N, K, dt=f16), T(n, dev=dev)),
                lambda n, dev="cuda:0": ops.linear_fp32(T(M, K), T(N, K), T(n, dev=dev)),
                lambda n, dev="cuda:0": ops.linear_fp8(x8.view(u8), w8.view(u8), 1.0, None, T(n, dev=dev)),
                lambda n, dev="cuda:0": ops.linear_int8_add_layernorm(x8, w8, 1.0, None, T(n, dev=dev), res, h, h, 1e-5),
                lambda n, dev="cuda:0": ops.linear_fp16_add_layernorm(T(M, K, dt=f16), T(N, K, dt=f16), T(n, dev=dev), res, h, h, 1e-5),
                lambda n, dev="cuda:0": ops.bias_gelu(T(M, N), T(n, dev=dev))],
            "gamma": [
                lambda n, dev="cuda:0": ops.layernorm(T(M, N), T(n, dev=dev), T(N)),
                lambda n, dev="cuda:0": ops.add_layernorm(res, res, T(n, dt=f16, dev=dev), h),
                lambda n, dev="cuda:0": ops.linear_int8_add_layernorm(x8, w8, 1.0, None, None, res, T(n, dt=f16, dev=dev), h, 1e-5),
                lambda n, dev="cuda:0": ops.embed_layernorm(ids, None, word, pos, typ, T(n, dt=f16, dev=dev), h, 1e-5, 16),
                lambda n, dev="cuda:0": ops.embed_layernorm_unpadded(ids, ids, None, word, pos, typ, T(n, dt=f16, dev=dev), h, 1e-5)],
            "beta": [lambda n, dev="cuda:0": ops.layernorm(T(M, N), T(N), T(n, dev=dev))],
            "type_ids": [lambda n, dev="cuda:0": ops.embed_layernorm(ids, T(n, dt=i32, dev=dev), word, pos, typ, h, h, 1e-5, 16)],
            "pos_packed": [lambda n, dev="cuda:0": ops.embed_layernorm_unpadded(ids, T(n, dt=i32, dev=dev), None, word, pos, typ, h, h, 1e-5)],
        }
        for name, fns in calls.items():
            for i, fn in enumerate(fns):
                with pytest.raises(RuntimeError, match=f"{name} must have (at least|one entry)"):
                    fn(2)
                with pytest.raises(RuntimeError, match=f"{name} must be on cuda:0"):
                    fn(2000, "cuda:1")
        for fn in (ops.linear_fp16, ops.linear_int8):
            dt = f16 if fn is ops.linear_fp16 else i8
            scale = () if fn is ops.linear_fp16 else (1.0,)
            with pytest.raises(RuntimeError, match="out must hold 4 x 768"):
                fn(T(M, K, dt=dt), T(N, K, dt=dt), *scale, out=T(M - 1, N, dt=f16), out_dtype=f16)
        with pytest.raises(RuntimeError, match="type must have at least 1536"):
            ops.embed_layernorm(ids, ids, word, pos, typ[:1], h, h, 1e-5, 16)


@pytest.mark.parametrize("name,dtype", [("wmma_matmul", "float16"), ("matmul_f32", "float32")])
def test_products_copy_each_strided_operand_once(monkeypatch, name, dtype):
    import torch
    from torch._subclasses.fake_tensor import FakeTensorMode
    from torch.utils._python_dispatch import TorchDispatchMode

    from zenith_b200 import ops

    copies = []

    class Count(TorchDispatchMode):
        def __torch_dispatch__(self, func, types, args=(), kwargs=None):
            if func is torch.ops.aten.clone.default:
                copies.append(tuple(args[0].shape))
            return func(*args, **(kwargs or {}))

    def no_device():
        raise InterruptedError

    monkeypatch.setattr(ops, "_stream", no_device)  # asked for after the copies, in front of the launch
    with FakeTensorMode():
        a, b = (torch.empty(s, dtype=getattr(torch, dtype), device="cuda:0").t() for s in ((64, 48), (32, 64)))
        with Count(), pytest.raises(InterruptedError):
            getattr(ops, name)(a, b)
    assert sorted(copies) == [(48, 64), (64, 32)]


def test_missing_extension_fails_loudly(monkeypatch, tmp_path):
    monkeypatch.setattr(_capi, "_lib", None)
    monkeypatch.setattr(_capi, "LIB_PATH", tmp_path / "absent.so")
    with pytest.raises(RuntimeError, match="no CPU or PyTorch fallback"):
        _capi.lib()
