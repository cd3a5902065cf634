"""The native host path (csrc/tq_host.cpp) against the general Python path of the same calls."""

import pytest
import torch

import tq_oracle as O

import turboquant as tq
from turboquant import cache

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(seed)


def _same(a, b):
    if isinstance(a, dict):
        return set(a) == set(b) and all(_same(a[k], b[k]) for k in a)
    if isinstance(a, (list, tuple)):
        return len(a) == len(b) and all(_same(x, y) for x, y in zip(a, b))
    if torch.is_tensor(a):
        return a.shape == b.shape and a.dtype == b.dtype and a.device == b.device and torch.equal(a, b)
    return a == b


@pytest.mark.parametrize("dim", [64, 96, 128])
@pytest.mark.parametrize("window", [0, 5, 128])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16, torch.float32])
def test_native_layer_path_equals_the_general_one(dim, window, dtype):
    codec = tq.TurboQuantV3(dim, key_bits=4, value_bits=3, residual_window=window, layer_idx=5, n_layers=32, device=DEV)
    base = O.synthetic_kv((2, 300, 3, dim), dtype, seed=dim + window).to(DEV)
    for keys in (base.transpose(1, 2), base.transpose(1, 2).contiguous(), base.transpose(1, 2)[:, 1:, 7:]):
        values = keys.flip(2)
        got, want = codec.compress_kv(keys, values), codec._compress_kv_general(keys, values)
        assert _same(got, want)
        assert got[0]["fp16"].data_ptr() == want[0]["fp16"].data_ptr()
        assert _same(codec.decompress_kv(*got), codec._decompress_kv_general(*want))
    mse = codec.key_compressor
    assert _same(mse.compress(keys), mse._compress_general(keys))
    assert _same(mse.decompress(got[0]["compressed"]), mse._decompress_general(got[0]["compressed"]))
    short = keys[:, :, :window]
    if window:
        ck, cv = codec.compress_kv(short, short)
        assert ck["compressed"] is None and codec.decompress_kv(ck, cv)[0] is ck["fp16"]


def test_native_layer_path_leaves_other_calls_to_the_general_one():
    codec = tq.TurboQuantV3(128, residual_window=4, layer_idx=5, device=DEV)
    x = O.synthetic_kv((1, 2, 40, 128), torch.float16, seed=1).to(DEV)
    columns = x.transpose(-1, -2).contiguous().transpose(-1, -2)              # last dimension not contiguous
    assert _same(codec.compress_kv(columns, columns)[0]["compressed"], codec.compress_kv(x, x)[0]["compressed"])
    mixed = codec.compress_kv(x, x.bfloat16())
    assert [t.dtype for t in codec.decompress_kv(*mixed)] == [torch.float16, torch.bfloat16]
    with pytest.raises(ValueError):
        codec.compress_kv(x[..., :64], x[..., :64])
    with pytest.raises(ValueError):
        codec.compress_kv(x.double(), x.double())
    grad = x.clone().requires_grad_()
    got, want = codec.compress_kv(grad, grad)[0], codec._compress_kv_general(grad, grad)[0]
    assert got["fp16"].requires_grad == want["fp16"].requires_grad and not got["compressed"]["vec_norms"].requires_grad


@pytest.mark.parametrize("window", [0, 16])
def test_native_cache_step_equals_the_general_one(window):
    L, shape = 5, (2, 3, 1, 128)
    made = []
    for native in (True, False):
        c = cache.V3Cache(key_bits=4, value_bits=2, residual_window=window, n_layers=L, initial_capacity=64)
        gen = _gen(11)
        outs = []
        for step in range(70):                                                # grows once, and S_new varies
            n = 3 if step % 9 == 4 else 1
            k, v = ([torch.randn(2, 3, n, 128, generator=gen, device=DEV).half() for _ in range(L)] for _ in range(2))
            fn = c.step if native else lambda a, b: c._step_general(a, b, True)
            outs.append([(x.clone(), y.clone()) for x, y in fn(k, v)])
        made.append((c, outs))
    (a, outs_a), (b, outs_b) = made
    assert _same(outs_a, outs_b)
    assert a.get_compression_info() == b.get_compression_info()
    for l in range(L):
        assert _same(a.packed_layer(l), b.packed_layer(l))
