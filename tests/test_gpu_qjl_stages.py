"""MSE + QJL compress where a CTA walks one, two or three tiles and the last one is ragged, against 64-bit sums.

Bounds: k_mse is an fp16 of a value right to 2^-20 of the vector's norm, and so is the residual (with wide codes a twentieth of the
vector), whose norm is an fp16 too.  A coordinate whose rotated value lies within 1e-6 of a threshold may take either index (its vector is left out), a sign whose
projection lies within 1e-5 of zero either sign."""

import math

import pytest
import torch

import turboquant as tq

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("packed", [False, True])
@pytest.mark.parametrize("bits", [2, 3, 4, 6])
@pytest.mark.parametrize("dim,n", [(128, 1), (128, 129), (256, 257), (256, 148 * 128 + 5), (128, 2 * 148 * 128 + 77), (128, 3 * 148 * 128 - 1)])
def test_stages_of_every_tile(dim, n, bits, packed):
    codec = tq.TurboQuantCompressorV2(dim, bits, seed=3, device=DEV)
    x = torch.randn(1, 1, n, dim, generator=torch.Generator(device=DEV).manual_seed(n + bits), device=DEV)
    x[..., :4] *= 10
    x = x.half()
    xd = x.double()
    norms = xd.norm(dim=-1)
    y = (xd / (norms + 1e-8)[..., None]) @ codec.Pi.double().T
    c = codec.centroids.double()
    edges = (c[1:] + c[:-1]) / 2
    idx = torch.searchsorted(edges, y)
    clear = ((y[..., None] - edges).abs().amin(dim=-1) > 1e-6).all(dim=-1)
    # thresholds lie 6 sigma / levels apart, sigma = dim ** -0.5: 256 coordinates of 5 bits meet 2e-6 / 0.012 of them, 4.4 % of the vectors
    assert float(clear.double().mean()) > 0.9
    mse = (c[idx] @ codec.Pi.double()) * norms[..., None]
    rest = xd - mse
    proj = rest @ codec.S.double().T
    sure = (proj.abs() > 1e-5 * norms[..., None]) & clear[..., None]
    out = codec.compress(x, packed=packed)
    if packed:
        mb = codec.mse_bits
        per = 8 // mb
        got = torch.stack([(out["mse_idx_bytes"].long() >> (mb * (per - 1 - i))) & (2 ** mb - 1) for i in range(per)], -1).flatten(-2)
        assert torch.equal(got[clear], idx[clear])
        signs = torch.stack([(out["sign_bits"].long() >> (7 - i)) & 1 for i in range(8)], -1).flatten(-2) * 2 - 1
        assert float(((out["vec_norms"].double() - norms) / norms).abs().max()) < dim * 2 ** -24
    else:
        k = out["k_mse"].double()
        bound = mse.abs() * 2 ** -11 + norms[..., None] * 2 ** -20 + 2 ** -24
        assert bool(((k - mse).abs() <= bound)[clear].all())
        signs = out["qjl_signs"].long()
    assert bool((signs == torch.where(proj >= 0, 1, -1))[sure].all())
    rn = rest.norm(dim=-1)
    err = (out["residual_norm"].double() - rn).abs()
    assert bool((err <= rn * 2 ** -11 + norms * 2 ** -20)[clear].all())
