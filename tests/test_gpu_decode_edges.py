"""Decode attention: block counts, windows without 16-byte rows, and the least scratch the entry point takes."""

import pytest
import torch

import tq_oracle as O

import turboquant as tq
from turboquant import _native as N

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(seed)


def _attend(codec, q, ck, cv):
    parts = []
    for side, comp in ((ck, codec.key_compressor), (cv, codec.val_compressor)):
        c = comp.centroids.double()
        B, H, S, D = side["compressed"]["shape"]
        idx = torch.from_numpy(O.unpack_indices(side["compressed"]["idx_bytes"].cpu().numpy().reshape(B * H * S, -1), comp.bits, D))
        back = (c[idx.to(DEV).long()] @ comp.Pi.double()).reshape(B, H, S, D) * side["compressed"]["vec_norms"].double().unsqueeze(-1)
        parts.append(torch.cat([back, side["fp16"].double()], dim=2))
    k, v = (p.repeat_interleave(q.shape[1] // p.shape[1], 1) for p in parts)
    return ((q.double() @ k.transpose(-1, -2)) * q.shape[-1] ** -0.5).softmax(-1) @ v


@pytest.mark.parametrize("window", [0, 1, 63, 65, 200])
@pytest.mark.parametrize("packed", [1, 255, 257, 5000])
@pytest.mark.parametrize("bits", [(4, 2), (8, 8)])
@pytest.mark.parametrize("dtype", [torch.float16, torch.float32])
def test_decode_attention_blocks_and_windows(window, packed, bits, dtype, monkeypatch):
    codec = tq.TurboQuantV3(128, key_bits=bits[0], value_bits=bits[1], residual_window=window, layer_idx=9, n_layers=32,
                            protected_layers=0, device=DEV)
    keys, vals = (O.synthetic_kv((1, 2, packed + window, 128), dtype, seed=s).to(DEV) for s in (packed, packed + 1))
    q = torch.randn(1, 6, 1, 128, generator=_gen(7), device=DEV)
    ck, cv = codec.compress_kv(keys, vals)
    want = _attend(codec, q, ck, cv)
    wide = codec.decode_attention(q, ck, cv)
    assert float((wide.double() - want).abs().max() / want.abs().max()) <= 1e-5
    # rows of 129 elements: no 16-byte loads from the window
    for side in (ck, cv):
        odd = torch.zeros(1, 2, window, 129, dtype=dtype, device=DEV)
        odd[..., 1:] = side["fp16"]
        side["fp16"] = odd[..., 1:]
    got = codec.decode_attention(q, ck, cv)
    assert float((got.double() - want).abs().max() / want.abs().max()) <= 1e-5
    # the least scratch that the entry point takes: one partial per 2048 keys
    L = N.lib()
    rows = 6
    least = (rows * 128 * 4 + 255) // 256 * 256 + rows * max(1, -(-packed // 2048)) * 130 * 4
    assert L.tq_decode_attention_workspace_bytes(1, 6, 1, packed) >= least
    monkeypatch.setattr(L, "tq_decode_attention_workspace_bytes", lambda *a: least)
    got = codec.decode_attention(q, ck, cv)
    assert float((got.double() - want).abs().max() / want.abs().max()) <= 1e-5
    monkeypatch.setattr(L, "tq_decode_attention_workspace_bytes", lambda *a: least - 4)
    with pytest.raises(ValueError):
        codec.decode_attention(q, ck, cv)


def test_a_refused_window_does_not_fail_the_next_call():
    """A window whose logits do not fit shared memory is refused before the launch; that error is this call's alone."""
    codec = tq.TurboQuantV3(128, key_bits=4, value_bits=2, residual_window=60000, layer_idx=9, n_layers=32, device=DEV)
    mse = codec.key_compressor
    small = O.synthetic_kv((1, 1, 300, 128), torch.float16, seed=1).to(DEV)
    want = mse.compress(small)["idx_bytes"]
    x = torch.zeros(1, 1, 60016, 128, dtype=torch.float16, device=DEV)
    ck, cv = codec.compress_kv(x, x)
    q = torch.ones(1, 1, 1, 128, dtype=torch.float16, device=DEV)
    with pytest.raises(RuntimeError):
        codec.decode_attention(q, ck, cv)
    assert torch.equal(mse.compress(small)["idx_bytes"], want)
    assert float((q + 1).sum()) == 256                                     # nor torch's own next launch


def test_back_to_back_calls_and_capture():
    """Scores and attention launch their kernels as a programmatic chain: calls in a row on one stream share scratch from the
    caching allocator, and a captured call replays the same."""
    codec = tq.TurboQuantV3(128, key_bits=4, value_bits=2, residual_window=16, layer_idx=9, n_layers=32, device=DEV)
    keys, vals = (O.synthetic_kv((1, 2, 3000, 128), torch.float16, seed=s).to(DEV) for s in (1, 2))
    ck, cv = codec.compress_kv(keys, vals)
    qs = [torch.randn(1, 8, 1, 128, generator=_gen(s), device=DEV).half() for s in range(40)]
    mse = codec.key_compressor

    def both(q):
        return (codec.decode_attention(q, ck, cv), *mse.attention_scores(q, ck["compressed"], scale=0.1, softmax=True))

    alone = []
    for q in qs:
        alone.append([t.clone() for t in both(q)])
        torch.cuda.synchronize()
    row = [both(q) for q in qs]
    torch.cuda.synchronize()
    for a, b in zip(alone, row):
        assert all(torch.equal(s, t) for s, t in zip(a, b))
    static = qs[0].clone()
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        both(static)
    torch.cuda.current_stream().wait_stream(side)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = both(static)
    for q, a in zip(qs[:5], alone):
        static.copy_(q)
        graph.replay()
        torch.cuda.synchronize()
        assert all(torch.equal(s, t) for s, t in zip(a, out))
