"""MSE + QJL kernels: buffers that start off a 32-byte boundary, and query counts around the operand's blocks."""

import ctypes as C
import math

import pytest
import torch

import tq_oracle as O

import turboquant as tq
from turboquant import _native as N

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(seed)


@pytest.mark.parametrize("d", [128, 256])
@pytest.mark.parametrize("packed", [False, True])
@pytest.mark.parametrize("rows", [1, 127, 129, 300])
def test_qjl_compress_off_a_32_byte_boundary(d, packed, rows):
    comp = tq.TurboQuantCompressorV2(d, 3, seed=9, device=DEV)
    buf = O.synthetic_kv((1, 1, rows + 1, d), torch.float16, seed=rows).to(DEV).reshape(-1)
    off = buf[8:8 + rows * d].view(1, 1, rows, d)
    assert off.data_ptr() % 32 == 16
    a, b = comp.compress(off, packed=packed), comp.compress(off.clone(), packed=packed)
    for key, want in b.items():
        if torch.is_tensor(want):
            assert torch.equal(a[key], want), key


@pytest.mark.parametrize("d", [128, 256])
@pytest.mark.parametrize("dtype", [torch.float32, torch.float16, torch.bfloat16])
@pytest.mark.parametrize("sq", [1, 31, 33, 64, 65, 130])
def test_qjl_scores_query_blocks(d, dtype, sq):
    """The query operand is built in blocks of 32 rows x 64 columns; rows past the end of a head are zero."""
    comp = tq.TurboQuantCompressorV2(d, 3, seed=9, device=DEV)
    keys = O.synthetic_kv((2, 3, 200, d), torch.float16, seed=sq).to(DEV)
    q = torch.randn(2, 3, sq, d, generator=_gen(sq), device=DEV).to(dtype)
    c = comp.compress(keys)
    got = comp.asymmetric_attention_scores(q, c)
    corr = math.sqrt(math.pi / 2) / d * c["residual_norm"].double().unsqueeze(-2)
    qd = q.double()
    want = qd @ c["k_mse"].double().transpose(-1, -2) + (qd @ comp.S.double().T) @ c["qjl_signs"].double().transpose(-1, -2) * corr
    assert float((got.double() - want).norm() / want.norm()) <= 1e-5
    assert N.lib().tq_last_device_status() == 0


@pytest.mark.parametrize("d", [64, 128, 256])
@pytest.mark.parametrize("sq", [1, 64, 100])
def test_scores_use_no_more_scratch_than_they_ask_for(d, sq, monkeypatch):
    """The operand images and the FP32 kernels' projections share one buffer; a guard behind it stays as it was."""
    comp = tq.TurboQuantCompressorV2(d, 3, seed=9, device=DEV)
    c = comp.compress(O.synthetic_kv((1, 3, 200, d), torch.float16, seed=sq).to(DEV))
    q = torch.randn(1, 3, sq, d, generator=_gen(sq), device=DEV)
    want = comp.asymmetric_attention_scores(q, c)
    wanted = N.lib().tq_qjl_scores_workspace_bytes(3, sq, d)
    units = 3 * -(-sq // 64)
    images = units * 8 * 64 * d + 1024 if d >= 128 else 0                   # four bytes (two pieces) of 2 D columns of 64 rows
    assert wanted == max(2 * 3 * sq * d * 4, images)
    made = []
    real = torch.empty

    def guarded(*size, **kw):
        if size == (max(wanted, 256),) and kw.get("dtype") is torch.uint8:
            made.append(torch.full((size[0] + 4096,), 0xA5, dtype=torch.uint8, device=DEV))
            return made[-1][:size[0]]
        return real(*size, **kw)
    monkeypatch.setattr(torch, "empty", guarded)
    got = comp.asymmetric_attention_scores(q, c)
    monkeypatch.undo()
    assert torch.equal(got, want) and len(made) == 1 and bool((made[0][-4096:] == 0xA5).all())


def test_one_query_needs_scratch_for_one_query():
    prod = tq.TurboQuantProd(128, 3, device=DEV)
    x = torch.randn(500, 128, generator=_gen(1), device=DEV)
    c = prod.quantize(x)
    L, y = N.lib(), torch.randn(1, 128, generator=_gen(2), device=DEV)
    want = prod.inner_product(y, c)
    out, ws = torch.empty(500, device=DEV), torch.full((2048 + 4096,), 0xA5, dtype=torch.uint8, device=DEV)

    def call(ny, n_bytes):
        return L.tq_prod_inner_product(y.data_ptr(), ny, c["mse_indices"].data_ptr(), c["qjl_signs"].data_ptr(), c["residual_norm"].data_ptr(),
                                       500, 128, c["qjl_signs"].shape[1], prod.mse.Pi.data_ptr(), prod.mse._cb.data_ptr(),
                                       prod._s_t.data_ptr(), out.data_ptr(), ws.data_ptr(), n_bytes, N.stream_ptr(DEV))
    assert call(1, 2048) == 0 and torch.equal(out, want) and bool((ws[2048:] == 0xA5).all())
    assert call(1, 2044) == -8 and call(500, 500 * 2048 - 4) == -8


def _guarded(n_bytes, off):
    """n_bytes on the device that start `off` bytes past a 32-byte boundary, and the buffer around them."""
    raw = torch.full((n_bytes + 128,), 0xA5, dtype=torch.uint8, device=DEV)
    start = 32 + (-raw.data_ptr()) % 32 + off
    return raw, start, raw[start:start + n_bytes]


@pytest.mark.parametrize("d", [128, 256])
@pytest.mark.parametrize("rows", [1, 127, 300])
def test_qjl_outputs_off_a_32_byte_boundary(d, rows):
    """k_mse and the signs may start on an odd multiple of 16 bytes: rows then leave as two 16-byte stores."""
    comp = tq.TurboQuantCompressorV2(d, 3, seed=9, device=DEV)
    x = O.synthetic_kv((1, 1, rows, d), torch.float16, seed=rows).to(DEV)
    L = N.lib()
    n_ws = L.tq_qjl_compress_workspace_bytes(rows, d)
    results = []
    for off in (0, 16):
        ws = torch.empty(n_ws, dtype=torch.uint8, device=DEV)
        raw_k, at_k, k = _guarded(rows * d * 2, off)
        raw_s, at_s, s = _guarded(rows * d, off)
        rnorm = torch.empty(rows, dtype=torch.float16, device=DEV)
        assert k.data_ptr() % 32 == off and s.data_ptr() % 32 == off
        job = N.QjlCompressJob(x=x.data_ptr(), x_dtype=N.F16, D=d, bits=comp.mse_bits, normalize=1, B=1, H=1, S=rows,
                               stride_b=rows * d, stride_h=rows * d, stride_s=d, rotation_t=comp.PiT.data_ptr(),
                               rotation=comp.Pi.data_ptr(), codebook=comp._cb.data_ptr(), qjl_t=comp._s_t.data_ptr(), M=d,
                               signs_dtype=0, rnorm_dtype=N.F16, idx_mode=N.IDX_U8, k_mse_out=k.data_ptr(), idx_out=None,
                               signs_out=s.data_ptr(), rnorm_out=rnorm.data_ptr(), workspace=ws.data_ptr(), workspace_bytes=n_ws,
                               vec_norms_out=None)
        N.check(L.tq_qjl_compress(C.byref(job), N.stream_ptr(DEV)), "tq_qjl_compress")
        for raw, at, out in ((raw_k, at_k, k), (raw_s, at_s, s)):
            assert bool((raw[:at] == 0xA5).all()) and bool((raw[at + out.numel():] == 0xA5).all())
        results.append((k.clone(), s.clone(), rnorm))
    assert all(torch.equal(a, b) for a, b in zip(*results))
    want = comp.compress(x)
    assert torch.equal(results[0][0].view(torch.float16).view(1, 1, rows, d), want["k_mse"])
    assert torch.equal(results[0][1].view(torch.int8).view(1, 1, rows, d), want["qjl_signs"])


@pytest.mark.parametrize("packed", [False, True])
@pytest.mark.parametrize("sq", [4, 40])
def test_back_to_back_mse_qjl_calls_and_capture(packed, sq):
    """Compress and scores launch their kernels as programmatic chains: calls in a row on one stream share scratch from the
    caching allocator, and a captured call replays the same."""
    comp = tq.TurboQuantCompressorV2(128, 3, seed=9, device=DEV)
    keys = [O.synthetic_kv((1, 2, 500, 128), torch.float16, seed=s).to(DEV) for s in range(20)]
    q = torch.randn(1, 2, sq, 128, generator=_gen(1), device=DEV).half()

    def both(x):
        c = comp.compress(x, packed=packed)
        return [v for v in c.values() if torch.is_tensor(v)] + [comp.asymmetric_attention_scores(q, c)]

    alone = []
    for x in keys:
        alone.append([t.clone() for t in both(x)])
        torch.cuda.synchronize()
    row = [both(x) for x in keys]
    torch.cuda.synchronize()
    for a, b in zip(alone, row):
        assert all(torch.equal(s, t) for s, t in zip(a, b))
    static = keys[0].clone()
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        both(static)
    torch.cuda.current_stream().wait_stream(side)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = both(static)
    for x, a in zip(keys[:5], alone):
        static.copy_(x)
        graph.replay()
        torch.cuda.synchronize()
        assert all(torch.equal(s, t) for s, t in zip(a, out))
    assert N.lib().tq_last_device_status() == 0
