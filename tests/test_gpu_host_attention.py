"""The native host path of the attention calls against the general Python path of the same calls: the same bits, and the
general path for everything that is not plain."""

import pytest
import torch

import turboquant as tq
from turboquant import _native as N
from turboquant import _ops, cache

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.fixture
def general(monkeypatch):
    def run(fn, *args, **kw):
        with monkeypatch.context() as m:
            m.setattr(N, "_host", N._GeneralPath())
            return fn(*args, **kw)
    return run


def _same(a, b):
    if isinstance(a, dict):
        return set(a) == set(b) and all(_same(a[k], b[k]) for k in a)
    if isinstance(a, (list, tuple)):
        return len(a) == len(b) and all(_same(x, y) for x, y in zip(a, b))
    if torch.is_tensor(a):
        return a.shape == b.shape and a.dtype == b.dtype and a.stride() == b.stride() and torch.equal(a, b)
    return a == b


@pytest.mark.parametrize("dtype", [torch.float16, torch.float32])
def test_scores_from_packed_keys(general, dtype):
    codec = tq.MSECompressor(128, 4, seed=1, device=DEV)
    packed = codec.compress(torch.randn(2, 2, 77, 128, device=DEV).half())
    q = torch.randn(2, 8, 3, 128, device=DEV).to(dtype)
    for softmax in (False, True):
        assert _same(codec.attention_scores(q, packed, scale=0.5, softmax=softmax), general(codec.attention_scores, q, packed, scale=0.5, softmax=softmax))
    H = N.host()
    plain = (q, packed["idx_bytes"], packed["vec_norms"], codec._pi_t, codec._cb, 4, 0.5, False)
    assert H.score_packed(*plain) is not None
    swap = lambda i, v: H.score_packed(*plain[:i], v, *plain[i + 1:])
    assert swap(0, q.transpose(1, 2).contiguous().transpose(1, 2)) is None and swap(0, q[:, :7]) is None
    assert swap(1, packed["idx_bytes"][..., :-1]) is None and swap(2, packed["vec_norms"].float()) is None
    assert swap(5, 9) is None and swap(5, 8) is None and swap(6, "1") is None and swap(7, 1) is None
    assert _same(codec.attention_scores(q.transpose(1, 2).contiguous().transpose(1, 2), packed), codec.attention_scores(q, packed))
    with pytest.raises(ValueError):
        codec.attention_scores(q[:, :7], packed)


@pytest.mark.parametrize("window", [0, 5])
def test_decode_attention(general, window):
    codec = tq.TurboQuantV3(128, key_bits=4, value_bits=2, residual_window=window, layer_idx=9, n_layers=32, protected_layers=0, device=DEV)
    x = torch.randn(2, 2, 90, 128, device=DEV).half()
    ck, cv = codec.compress_kv(x, x.flip(2).contiguous())
    q = torch.randn(2, 8, 1, 128, device=DEV).half()
    assert _same(codec.decode_attention(q, ck, cv), general(codec.decode_attention, q, ck, cv))
    H = N.host()
    args = (q, ck["compressed"], cv["compressed"], codec.key_compressor, codec.val_compressor, ck["fp16"], cv["fp16"], 0.1)
    assert H.decode_attention(*args) is not None
    assert H.decode_attention(*args[:1], None, *args[2:]) is None                     # nothing packed: the general path
    assert H.decode_attention(q[:, :7], *args[1:]) is None
    assert H.decode_attention(*args[:2], {**cv["compressed"], "idx_bytes": cv["compressed"]["idx_bytes"][:, :, 1:]}, *args[3:]) is None
    if window:
        assert H.decode_attention(*args[:6], cv["fp16"].float(), 0.1) is None
    with pytest.raises(ValueError):
        codec.decode_attention(q[:, :7], ck, cv)


@pytest.mark.parametrize("dim", [64, 128])
def test_mse_qjl(general, dim):
    codec = tq.TurboQuantCompressorV2(dim, 3, seed=1, device=DEV)
    x, q = torch.randn(2, 3, 70, dim, device=DEV).half(), torch.randn(2, 3, 4, dim, device=DEV).half()
    forms = [False] + [True] * (dim == 128)
    for packed in forms:
        got = codec.compress(x, packed=packed)
        assert _same(got, general(codec.compress, x, packed=packed))
        assert _same(codec.asymmetric_attention_scores(q, got), general(codec.asymmetric_attention_scores, q, got))
    every_other = codec.compress(x[:, :, ::2], packed=False)                          # strided: the general path or its kernels
    assert _same(every_other, general(codec.compress, x[:, :, ::2], packed=False))
    grad = x.clone().requires_grad_()
    assert not codec.compress(grad)["k_mse"].requires_grad


def test_views_of_a_step_are_views_of_the_buffers():
    c = cache.V3Cache(key_bits=4, value_bits=2, residual_window=4, n_layers=2, initial_capacity=32)
    for _ in range(8):
        out = c.step(*([torch.randn(1, 2, 1, 128, device=DEV).half() for _ in range(2)] for _ in range(2)))
    for l, pair in enumerate(out):
        for view, buf in zip(pair, (c._layers[l].k, c._layers[l].v)):
            want = buf.narrow(2, 0, 8)
            assert view.data_ptr() == want.data_ptr() and view.shape == want.shape and view.stride() == want.stride()
            assert view._is_view() and view._version == buf._version
            view[0, 0, 0, 0] = 1
            assert view._version == buf._version and float(buf[0, 0, 0, 0]) == 1
