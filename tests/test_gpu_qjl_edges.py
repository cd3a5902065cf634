"""MSE + QJL kernels: buffers that start off a 32-byte boundary, and query counts around the operand's blocks."""

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
