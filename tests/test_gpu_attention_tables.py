"""Packed-key scores and decode attention at the edges of their key blocks, for every code width and both numbers of query
rows per pass, against 64-bit sums of the same packed bytes.

Bound: centroids and rotated queries travel as two fp16 pieces each (off by 2^-22 of the value), products add up in fp32
over 128 coordinates: |error| <= (2 * 2^-22 + 128 * 2^-24) |q| |k| < 1e-5 |q| |k| for a logit."""

import ctypes as C

import pytest
import torch

import turboquant as tq
from turboquant import _native as N
from turboquant import _ops

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _packed(comp, shape, seed):
    """Any bytes at all (unused bits of 3- and 5- to 7-bit codes included) and their 64-bit reconstruction."""
    g = torch.Generator(device=DEV).manual_seed(seed)
    per = 8 // comp.bits
    idx = torch.randint(0, 256, shape[:3] + (128 // per,), generator=g, device=DEV, dtype=torch.uint8)
    norms = (torch.rand(shape[:3], generator=g, device=DEV) * 10 + 1).half()
    fields = [(idx.long() >> (comp.bits * (per - 1 - i))) & (2 ** comp.bits - 1) for i in range(per)]
    levels = comp.centroids.double()[torch.stack(fields, -1).flatten(-2)]
    return {"idx_bytes": idx, "vec_norms": norms, "shape": shape, "idx_pad": 0}, (levels @ comp.Pi.double()) * norms.double()[..., None]


def _logits(q, k, rep):
    return torch.einsum("bhrqd,bhkd->bhrqk", q.double().unflatten(1, (-1, rep)), k).flatten(1, 2) * 0.25


@pytest.mark.parametrize("rows", [(1, 1), (4, 1), (3, 2), (8, 1)])
@pytest.mark.parametrize("bits", range(1, 9))
def test_scores_at_block_edges(bits, rows):
    rep, sq = rows
    comp = tq.MSECompressor(128, bits, seed=5, device=DEV)
    for sk in (1, 15, 16, 17, 127, 129, 300):
        q = torch.randn(2, 2 * rep, sq, 128, generator=torch.Generator().manual_seed(sk)).to(DEV)
        packed, k = _packed(comp, (2, 2, sk, 128), 100 * bits + sk)
        logits, probs = comp.attention_scores(q, packed, scale=0.25, softmax=True)
        want = _logits(q, k, rep)
        bound = 1e-5 * 0.25 * float(q.double().norm(dim=-1).max() * k.norm(dim=-1).max())
        assert float((logits - want).abs().max()) <= bound
        # a probability's relative error is that of its logit, and of the largest; the exponentials add 1e-6
        assert float((probs - want.softmax(-1)).abs().max()) <= 3 * bound + 1e-5


def test_scores_with_the_least_scratch():
    """Blocks of 1024 keys at least, as much as callers brought before: the same numbers."""
    comp = tq.MSECompressor(128, 4, seed=5, device=DEV)
    q = torch.randn(1, 8, 1, 128, generator=torch.Generator().manual_seed(1)).to(DEV)
    packed, k = _packed(comp, (1, 2, 5000, 128), 7)
    want, want_p = comp.attention_scores(q, packed, scale=0.25, softmax=True)
    rows, q_bytes = 8, 8 * 128 * 4
    least = q_bytes + rows * 5 * 8
    ws = torch.full((least + 4096,), 171, dtype=torch.uint8, device=DEV)
    logits, probs = torch.empty_like(want), torch.empty_like(want)
    job = N.ScoreJob(q=q.data_ptr(), q_dtype=N.dtype_code(q), D=128, bits=4, reserved=0, B=1, Hq=8, Sq=1, Hkv=2, Sk=5000,
                     idx_bytes=packed["idx_bytes"].data_ptr(), norms=packed["vec_norms"].data_ptr(), rotation_t=comp._pi_t.data_ptr(),
                     codebook=comp._cb.data_ptr(), scale=0.25, reserved2=0, logits=logits.data_ptr(), probs=probs.data_ptr(),
                     workspace=ws.data_ptr(), workspace_bytes=least)
    N.check(N.lib().tq_score_packed(C.byref(job), N.stream_ptr(q.device)), "tq_score_packed")
    job.workspace_bytes = least - 1
    assert N.lib().tq_score_packed(C.byref(job), N.stream_ptr(q.device)) != 0
    assert torch.equal(logits, want)                                      # one key's sum does not depend on its block
    assert torch.allclose(probs, want_p, rtol=1e-5, atol=1e-9)            # the sum of 5000 exponentials in another order
    assert bool((ws[least:] == 171).all())


@pytest.mark.parametrize("bits", [(1, 1), (2, 2), (3, 3), (4, 2), (4, 4), (5, 3), (6, 4), (7, 7), (8, 8), (2, 8), (8, 1)])
def test_decode_attention_at_block_edges(bits):
    codec = tq.TurboQuantV3(128, key_bits=bits[0], value_bits=bits[1], residual_window=0, layer_idx=3, n_layers=36,
                            protected_layers=0, device=DEV)
    for rep in (1, 5):
        for sk in (1, 15, 17, 31, 33, 255, 257, 700):
            q = torch.randn(1, 2 * rep, 1, 128, generator=torch.Generator().manual_seed(sk)).to(DEV)
            pk, k = _packed(codec.key_compressor, (1, 2, sk, 128), sk)
            pv, v = _packed(codec.val_compressor, (1, 2, sk, 128), sk + 1)
            empty = torch.empty(1, 2, 0, 128, dtype=torch.float16, device=DEV)
            ck, cv = ({"compressed": c, "fp16": empty, "shape": c["shape"], "split_at": sk} for c in (pk, pv))
            out = codec.decode_attention(q, ck, cv, scale=0.25)
            p = _logits(q, k, rep).softmax(-1)
            want = torch.einsum("bhrqk,bhkd->bhrqd", p.unflatten(1, (-1, rep)), v).flatten(1, 2)
            # a logit's error moves every weight by that share, and so the sum by that share of the largest value
            bound = 1e-5 * 0.25 * float(q.double().norm(dim=-1).max() * k.norm(dim=-1).max())
            assert float((out - want).abs().max()) <= (2 * bound + 1e-5) * float(v.norm(dim=-1).max())
