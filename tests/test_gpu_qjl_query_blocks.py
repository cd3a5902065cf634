"""MSE + QJL scores around the line between 16 and 64 queries per pass, keys around the edge of a tile, against 64-bit sums.

Bound: the query operand is two fp16 pieces (off by 2^-22), its projection an fp32 chain of `dim` terms, the products add up
in fp32 over 2 dim coordinates: |error| <= (2^-21 + 3 dim 2^-24) |operands|, below 1e-4 of the largest score's terms."""

import math

import pytest
import torch

import turboquant as tq

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("dim", [128, 256])
@pytest.mark.parametrize("queries", [1, 15, 16, 17, 63, 65])
def test_scores_around_the_query_blocks(dim, queries):
    codec = tq.TurboQuantCompressorV2(dim, 3, seed=4, device=DEV)
    for keys in (1, 127, 128, 300, 1025):
        g = torch.Generator(device=DEV).manual_seed(keys)
        x = torch.randn(2, 3, keys, dim, generator=g, device=DEV).half()
        q = torch.randn(2, 3, queries, dim, generator=g, device=DEV).half()
        c = codec.compress(x)
        got = codec.asymmetric_attention_scores(q, c)
        k, s, r = c["k_mse"].double(), c["qjl_signs"].double(), c["residual_norm"].double()
        proj = q.double() @ codec.S.double().T * (math.sqrt(math.pi / 2) / dim)
        want = q.double() @ k.transpose(-1, -2) + proj @ s.transpose(-1, -2) * r[:, :, None]
        size = (q.double().abs() @ k.abs().transpose(-1, -2) + proj.abs().sum(-1, keepdim=True) * r[:, :, None])
        assert bool(((got - want).abs() <= (2 ** -21 + 3 * dim * 2 ** -24) * size).all())
