"""The native host path (csrc/tq_host.cpp) against the general Python path of the same calls."""

import pytest
import torch

import tq_oracle as O

import turboquant as tq
from turboquant import _native as N
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


# ------------------------------------------------------------------ that the native form is what ran
@pytest.fixture
def general(monkeypatch):
    """Runs a call with the extension out of the way."""
    def run(fn):
        with monkeypatch.context() as m:
            m.setattr(N, "_host", N._GeneralPath())
            return fn()
    return run


def _taken(fn, *args):
    out = fn(*args)
    assert out is not None, fn.__name__
    return out


def test_plain_layer_calls_are_taken():
    H = N.host()
    codec = tq.TurboQuantV3(128, key_bits=4, value_bits=3, residual_window=5, layer_idx=5, device=DEV)
    x = O.synthetic_kv((2, 3, 100, 128), torch.float16, seed=1).to(DEV)
    kc, vc = codec.key_compressor, codec.val_compressor
    for keys in (x, x.transpose(1, 2).contiguous().transpose(1, 2), x[:, 1:, 7:]):
        ck, cv = _taken(H.compress_kv, kc, vc, keys, keys, 5, codec.compress_jobs)
        assert _same((ck, cv), codec._compress_kv_general(keys, keys))
        assert _same(_taken(H.decompress_kv, kc, vc, ck, cv, codec.decompress_jobs), codec._decompress_kv_general(ck, cv))
        packed = _taken(H.compress, kc, keys)
        assert _same(packed, kc._compress_general(keys))
        assert _same(_taken(H.decompress, kc, packed), kc._decompress_general(packed))
    columns = x.transpose(-1, -2).contiguous().transpose(-1, -2)
    for odd in (columns, x.double(), x.cpu(), x[..., :64]):                 # what the general path copies or refuses
        assert H.compress(kc, odd) is None and H.compress_kv(kc, vc, odd, odd, 5, codec.compress_jobs) is None
    assert H.compress_kv(kc, vc, x, x, 100, codec.compress_jobs) is None                         # nothing leaves the window
    short = {**packed, "idx_bytes": packed["idx_bytes"][..., :-1].contiguous()}
    assert H.decompress(kc, short) is None and H.decompress(kc, {**packed, "vec_norms": packed["vec_norms"].float()}) is None


def test_plain_cache_steps_are_taken():
    L = 3
    c = cache.V3Cache(key_bits=4, value_bits=2, residual_window=8, n_layers=L, initial_capacity=64)
    gen = _gen(3)
    for step in range(20):
        k, v = ([torch.randn(1, 2, 1, 128, generator=gen, device=DEV).half() for _ in range(L)] for _ in range(2))
        c.step(k, v)
    assert c._native_plan is not None and c._native_plan[0] is not None
    assert len(c._step_log) >= 10                                           # twelve tokens left the window, the first steps made the layers
    assert N.host().step(c._native_plan[0], c._native_plan[2], [t.float() for t in k], v, True, c._step_log) is None
    assert c.get_compression_info() == "12 compressed, 8 fp16, 20 total"


def test_mixed_updates_and_steps_keep_token_order():
    L = 2
    made = []
    for native in (True, False):
        c = cache.V3Cache(key_bits=4, value_bits=2, residual_window=4, n_layers=L, initial_capacity=64)
        gen = _gen(5)
        for step in range(30):
            k, v = ([torch.randn(1, 2, 1, 128, generator=gen, device=DEV).half() for _ in range(L)] for _ in range(2))
            if step % 7 == 3:
                for l in range(L):
                    c.update(k[l], v[l], l)
            elif native:
                c.step(k, v)
            else:
                c._step_general(k, v, True)
        made.append([c.packed_layer(l) for l in range(L)])
        assert (len(c._step_log) > 0) == native
        again = cache.V3Cache.from_cache_state(c.cache_state())
        assert _same(made[-1], [again.packed_layer(l) for l in range(L)])
    assert _same(made[0], made[1])


@pytest.mark.parametrize("d", [64, 96, 128])
def test_plain_first_generation_calls_are_taken(d, general):
    H = N.host()
    x = torch.randn(50, d, generator=_gen(d), device=DEV)
    x = x / x.norm(dim=-1, keepdim=True)
    mse, prod = tq.TurboQuantMSE(d, 3, device=DEV), tq.TurboQuantProd(d, 3, device=DEV)
    idx = _taken(H.quantize_rows, x, mse._pi_t, mse._cb, 3, d)
    assert _same(idx, general(lambda: mse.quantize(x)))
    assert _same(_taken(H.dequantize_rows, idx, mse.Pi, mse._cb, 3, d), general(lambda: mse.dequantize(idx)))
    assert H.quantize_rows(x.t().contiguous().t(), mse._pi_t, mse._cb, 3, d) is None
    assert H.dequantize_rows(idx.int(), mse.Pi, mse._cb, 3, d) is None
    c = general(lambda: prod.quantize(x))
    got = _taken(H.qjl_compress, x.view(1, 1, 50, d), prod.mse.Pi, prod.mse._pi_t, prod.mse._cb, prod._s_t, prod.mse_bits, 2)
    assert _same(tuple(got), (c["mse_indices"], c["qjl_signs"], c["residual_norm"]))
    for y in (x, x[:1]):
        ip = _taken(H.prod_inner, y, *got, prod.mse.Pi, prod.mse._cb, prod._s_t)
        assert _same(ip, general(lambda: prod.inner_product(y if y.shape[0] > 1 else y[0], c)))
    assert H.prod_inner(x[:2], *got, prod.mse.Pi, prod.mse._cb, prod._s_t) is None


@pytest.mark.parametrize("d", [64, 128, 256])
@pytest.mark.parametrize("packed", [False, True])
def test_plain_mse_qjl_calls_are_taken(d, packed, general):
    comp = tq.TurboQuantCompressorV2(d, 3, seed=9, device=DEV)
    x = O.synthetic_kv((1, 2, 70, d), torch.float16, seed=d).to(DEV)
    args = (comp.Pi, comp.PiT, comp._cb, comp._s_t, comp.mse_bits, int(packed))
    if packed and d == 64:
        assert N.host().qjl_compress(x, *args) is None                      # no tensor-core path: packed in a second pass
    else:
        _taken(N.host().qjl_compress, x, *args)
    assert _same(comp.compress(x, packed=packed), general(lambda: comp.compress(x, packed=packed)))
    assert N.host().qjl_compress(x[:, :, :0], *args) is None


# ------------------------------------------------------------------ codecs with job methods of their own
class _OwnJobs(tq.MSECompressor):
    """Counts what it is asked, and packs zeros."""

    def compress_job(self, states):
        self.asked = getattr(self, "asked", 0) + 1
        return super().compress_job(torch.zeros_like(states))

    def decompress_job(self, compressed, out):
        self.asked = getattr(self, "asked", 0) + 1
        return super().decompress_job({**compressed, "vec_norms": torch.zeros_like(compressed["vec_norms"])}, out)


class _OwnLayerJobs(tq.TurboQuantV3):
    def compress_jobs(self, keys, values):
        return super().compress_jobs(torch.zeros_like(keys), values)

    def decompress_jobs(self, compressed_k, compressed_v):
        jobs, outs, keep = super().decompress_jobs(compressed_k, compressed_v)
        return jobs, outs[::-1], keep


def _zeros(packed):
    return bool((packed["vec_norms"] == 0).all())


def test_a_subclass_that_overrides_its_jobs_is_asked():
    x = O.synthetic_kv((1, 2, 40, 128), torch.float16, seed=1).to(DEV)
    comp = _OwnJobs(128, 4, seed=1, device=DEV)
    assert _zeros(comp.compress(x)) and comp.asked == 1
    packed = tq.MSECompressor(128, 4, seed=1, device=DEV).compress(x)
    assert not comp.decompress(packed).any() and comp.asked == 2
    layer = _OwnLayerJobs(128, residual_window=8, layer_idx=9, n_layers=32, device=DEV)
    ck, cv = layer.compress_kv(x, x)
    assert _zeros(ck["compressed"]) and not _zeros(cv["compressed"])
    values, keys = layer.decompress_kv(ck, cv)
    assert not keys[:, :, :32].any() and values[:, :, :32].any()


@pytest.mark.parametrize("side", ["key_compressor", "val_compressor"])
@pytest.mark.parametrize("how", ["subclass", "object", "patch"])
def test_a_layer_with_such_a_codec_asks_it(side, how, monkeypatch):
    x = O.synthetic_kv((1, 2, 40, 128), torch.float16, seed=1).to(DEV)
    layer = tq.TurboQuantV3(128, residual_window=0, layer_idx=9, n_layers=32, device=DEV)
    plain = layer.compress_kv(x, x)
    comp = getattr(layer, side)
    if how == "subclass":
        setattr(layer, side, _OwnJobs(128, comp.bits, seed=1, device=DEV))
    elif how == "object":
        own = comp.compress_job
        comp.compress_job = lambda states: own(torch.zeros_like(states))
        back = comp.decompress_job
        comp.decompress_job = lambda packed, out: back({**packed, "vec_norms": torch.zeros_like(packed["vec_norms"])}, out)
    else:
        for name in ("compress_job", "decompress_job"):
            monkeypatch.setattr(tq.MSECompressor, name, _patched(name, comp))
    zeros = [_zeros(c["compressed"]) for c in layer.compress_kv(x, x)]
    assert zeros == [side == "key_compressor", side == "val_compressor"]
    assert [not t.any() for t in layer.decompress_kv(*plain)] == zeros


def _patched(name, which):
    own = getattr(tq.MSECompressor, name)
    if name == "compress_job":
        return lambda self, states: own(self, torch.zeros_like(states) if self is which else states)
    return lambda self, packed, out: own(self, {**packed, "vec_norms": packed["vec_norms"] * (0 if self is which else 1)}, out)
