"""Calls of few vectors (csrc/tq_few.cu) against the FP32 kernels, whose chain of operations per value they share."""

import os

import pytest
import torch

import tq_oracle as O

import turboquant as tq
from turboquant import _native as N
from turboquant import _ops

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _simt(fn):
    os.environ["TQ_FORCE_SIMT"] = "1"
    try:
        return fn()
    finally:
        os.environ.pop("TQ_FORCE_SIMT", None)


def _equal(a, b):
    return torch.equal(a, b) or torch.equal(a.isnan(), b.isnan()) and torch.equal(a.nan_to_num(), b.nan_to_num())


@pytest.mark.parametrize("dim", [64, 128])
@pytest.mark.parametrize("dtype", [torch.float32, torch.float16, torch.bfloat16])
@pytest.mark.parametrize("bits", [1, 2, 3, 4, 5, 6, 7, 8])
@pytest.mark.parametrize("heads,seq", [(1, 1), (3, 1), (5, 7), (40, 16)])
def test_few_vectors_equal_the_fp32_kernels(dim, dtype, bits, heads, seq):
    base = O.synthetic_kv((2, heads, seq + 3, dim + 8), dtype, seed=bits + seq).to(DEV)
    x = base[:, :, 2:seq + 2, 3:dim + 3]                                   # strided, rows off their 16-byte boundary
    if seq > 1:
        base[0, 0, 3, 5] = float("nan")
        base[1, heads - 1, 2, 7] = float("inf")
        base[0, heads - 1, 4] = 0
    comp = tq.MSECompressor(dim, bits, seed=4, device=DEV)
    got, want = comp.compress(x), _simt(lambda: comp.compress(x))
    assert torch.equal(got["idx_bytes"], want["idx_bytes"]) and _equal(got["vec_norms"], want["vec_norms"])
    for out_dtype in (torch.float32, torch.float16, torch.bfloat16):
        for shift in (0, 1):                                               # 16-byte rows, and rows off their boundary
            outs = []
            for run in (lambda f: f(), _simt):
                out = torch.full((2, heads, seq + 2, dim + 8), -3.0, dtype=out_dtype, device=DEV)
                view = out[:, :, 1:seq + 1, shift:dim + shift]
                job, _keep = comp.decompress_job(want, view)
                run(lambda: _ops.run_dequantize([job], DEV))
                outs.append(out)
            assert _equal(outs[0], outs[1])


@pytest.mark.parametrize("mode,dtype", [(N.IDX_U8, torch.uint8), (N.IDX_I64, torch.int64)])
@pytest.mark.parametrize("normalize", [False, True])
def test_few_vectors_other_layouts(mode, dtype, normalize):
    comp = tq.MSECompressor(128, 3, seed=4, device=DEV)
    x = torch.randn(1, 2, 9, 128, generator=torch.Generator(device=DEV).manual_seed(1), device=DEV)
    x = x / x.norm(dim=-1, keepdim=True)
    done = []
    for run in (lambda f: f(), _simt):
        job, idx, norms, _keep = _ops.quantize_job(x, comp._pi_t, comp._cb, 3, normalize, mode)
        run(lambda: _ops.run_quantize([job], DEV))
        out = torch.empty(1, 2, 9, 128, device=DEV)
        back, _keep2 = _ops.dequantize_job(idx, norms, (1, 2, 9, 128), comp.Pi, comp._cb, 3, mode, out)
        run(lambda: _ops.run_dequantize([back], DEV))
        done.append((idx, norms, out))
    (ia, na, oa), (ib, nb, ob) = done
    assert ia.dtype == dtype and torch.equal(ia, ib) and torch.equal(oa, ob)
    assert na is None and nb is None or torch.equal(na, nb)


@pytest.mark.parametrize("jobs", [2, 8, 9, 96, 97, 200])
def test_many_jobs_of_few_vectors(jobs):
    comps = [tq.MSECompressor(128, 2 + i % 7, seed=i, device=DEV) for i in range(min(jobs, 12))]
    x = [torch.randn(1, 1 + i % 3, 1 + i % 5, 128, generator=torch.Generator(device=DEV).manual_seed(i), device=DEV).half() for i in range(jobs)]

    def run():
        made = [comps[i % len(comps)].compress_job(x[i]) for i in range(jobs)]
        _ops.run_quantize([m[0] for m in made], DEV)
        outs, back = [], []
        for i, m in enumerate(made):
            outs.append(torch.empty_like(x[i]))
            back.append(comps[i % len(comps)].decompress_job(m[1], outs[i]))
        _ops.run_dequantize([b[0] for b in back], DEV)
        return [(m[1]["idx_bytes"], m[1]["vec_norms"], o) for m, o in zip(made, outs)]

    for a, b in zip(run(), _simt(run)):
        assert all(torch.equal(s, t) for s, t in zip(a, b))


def _round_trip(comp, x, room):
    """One call over all of x and back into 16-bit rows; `room` more elements per row keep the rows off 16-byte boundaries."""
    packed = [comp.compress_job(t) for t in x]
    _ops.run_quantize([p[0] for p in packed], DEV)
    outs, back = [], []
    for t, p, r in zip(x, packed, room):
        outs.append(torch.empty(*t.shape[:3], t.shape[3] + r, dtype=t.dtype, device=DEV)[..., r // 2:r // 2 + t.shape[3]])
        back.append(comp.decompress_job(p[1], outs[-1]))
    _ops.run_dequantize([b[0] for b in back], DEV)
    return [(p[1]["idx_bytes"], p[1]["vec_norms"], o) for p, o in zip(packed, outs)]


@pytest.mark.parametrize("dim", [64, 128])
@pytest.mark.parametrize("slabs", [(3000,), (1500, 1500), (2999, 1), (1, 2999)])
@pytest.mark.parametrize("odd", [None, "first", "last"])
def test_the_limit_counts_vectors_and_not_jobs(dim, slabs, odd):
    """3000 tokens of a slab each run here as one job or as two, alone or before or behind 900 vectors that only the FP32
    kernels take.  The tensor-core kernels' 16-bit reconstruction would not be the FP32 kernels'."""
    comp = tq.MSECompressor(dim, 4, seed=4, device=DEV)
    gen = torch.Generator(device=DEV).manual_seed(1)
    x = [torch.randn(1, n, 1, dim, generator=gen, device=DEV).half() for n in slabs]
    room = [0] * len(x)
    if odd is not None:
        at = 0 if odd == "first" else len(x)
        x.insert(at, torch.randn(1, 60, 15, dim + 6, generator=gen, device=DEV).half()[..., 3:dim + 3])
        room.insert(at, 6)
    for a, b in zip(_round_trip(comp, x, room), _simt(lambda: _round_trip(comp, x, room))):
        assert all(torch.equal(s, t) for s, t in zip(a, b))


@pytest.mark.parametrize("jobs", [1, 2, 8])
def test_fuller_tiles_stay_on_the_tensor_cores(jobs):
    """Slabs of 16 tokens, 4096 vectors in all at head_dim 128: the same values as in a long call of the same tokens."""
    comp = tq.MSECompressor(128, 4, seed=4, device=DEV)
    long = torch.randn(1, 256, 160, 128, generator=torch.Generator(device=DEV).manual_seed(1), device=DEV).half()
    (idx, norms, back), = _round_trip(comp, [long], [0])
    x = [t.contiguous() for t in long[:, :, :16].chunk(jobs, dim=1)]
    got = _round_trip(comp, x, [0] * jobs)
    assert torch.equal(torch.cat([g[0] for g in got], 1), idx[:, :, :16]) and torch.equal(torch.cat([g[1] for g in got], 1), norms[:, :, :16])
    assert torch.equal(torch.cat([g[2] for g in got], 1), back[:, :, :16])
