"""The FP32 kernels at the edges of their tiles, and the one-query inner product."""

import math

import pytest
import torch

import tq_oracle as O

import turboquant as tq
from turboquant import _native as N
from turboquant import _ops

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(seed)


@pytest.mark.parametrize("d", [33, 64, 100, 128, 200, 256])
@pytest.mark.parametrize("rows", [1, 31, 32, 33, 97])
def test_fp32_results_do_not_depend_on_the_tile_size(d, rows):
    """Many vectors run in tiles of 64, few in tiles of 32, with the same chain of operations per output: the first rows of a
    large call are bit for bit those of a small one, and match 64-bit sums."""
    many = 64 * 2 * 160 + 5
    x = torch.randn(1, 1, many, d, generator=_gen(d + rows), device=DEV)
    comp = tq.MSECompressor(d, 4, seed=3, device=DEV)
    big, small = comp.compress(x), comp.compress(x[:, :, :rows])
    assert torch.equal(big["idx_bytes"][:, :, :rows], small["idx_bytes"])
    assert torch.equal(big["vec_norms"][:, :, :rows], small["vec_norms"])
    back_big, back_small = _simt_decompress(comp, big), _simt_decompress(comp, small)
    assert torch.equal(back_big[:, :, :rows], back_small)
    # every centroid is the nearest one, up to the rounding of the fp32 chains
    unit = x[0, 0, :rows].double() / x[0, 0, :rows].double().norm(dim=-1, keepdim=True)
    y, c = unit @ comp.Pi.double().T, comp.centroids.double()
    idx = torch.from_numpy(O.unpack_indices(small["idx_bytes"].cpu().numpy().reshape(rows, -1), 4, d)).to(DEV).long()
    assert float(((y - c[idx]).abs() - (y.unsqueeze(-1) - c).abs().amin(-1)).max()) <= 1e-6
    want = (c[idx] @ comp.Pi.double()) * small["vec_norms"][0, 0].double().unsqueeze(-1)
    assert float((back_small[0, 0].double() - want).norm() / want.norm()) <= 1e-6


def _simt_decompress(comp, packed):
    B, H, S, D = packed["shape"]
    out = torch.empty((B, H, S, D), dtype=torch.float32, device=DEV)
    job, _keep = _ops.dequantize_job(packed["idx_bytes"], packed["vec_norms"], packed["shape"], comp.Pi, comp._cb, comp.bits,
                                     N.IDX_PACKED, out, image=None)
    _ops.run_dequantize([job], DEV)
    return out


@pytest.mark.parametrize("d,m", [(64, 64), (128, 128), (100, 37), (256, 250)])
@pytest.mark.parametrize("rows", [1, 33, 700])
def test_one_query_against_every_vector(d, m, rows):
    """The one-query form rotates the query; the paired form rotates every vector back."""
    p = tq.TurboQuantProd(d, 3, qjl_dim=m, seed=5, device=DEV)
    x = torch.randn(rows, d, generator=_gen(rows), device=DEV)
    y = torch.randn(1, d, generator=_gen(rows + 1), device=DEV)
    c = p.quantize(x / x.norm(dim=-1, keepdim=True))
    one = p.inner_product(y, c)
    pairs = torch.cat([y, y.new_zeros(1, d)]).repeat_interleave(rows, 0)[:rows].contiguous() if rows > 1 else y
    paired = p.inner_product(pairs, c)
    xhat = p.mse.centroids.double()[c["mse_indices"]] @ p.mse.Pi.double()
    want = xhat @ y[0].double() + math.sqrt(math.pi / 2) / m * c["residual_norm"].double() * (c["qjl_signs"].double() @ (p.S.double() @ y[0].double()))
    scale = float(want.abs().max()) + 1e-3
    assert float((one.double() - want).abs().max()) <= 1e-5 * scale
    assert float((paired.double() - want).abs().max()) <= 1e-5 * scale
