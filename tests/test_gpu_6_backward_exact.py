"""Tensor-core backward of the calls that carry score modifiers, a dense bias or the latent head shape.

Its P and dS enter the products as 16 + 16 bits, so its 16-bit gradients may differ from those of the exact-fp32
CUDA-core kernels (same inputs, same saved o and lse) by the rounding of the result only: one unit in the last
place of an element, 2^-8 (bf16) or 2^-11 (fp16) of it, hence at most that of the norm.  The bias gradient is fp32;
its error is that of the scores and of dP, sums of D products (2^-24 sqrt(D) each, doubled for the unit's
truncation), times the cancellation in dP - delta: 1e-4 of the norm leaves a factor of ten.
"""

import math

import pytest
import torch

from probjax_b200 import attention as A
from probjax_b200 import masks as M
from _gpu_util import dev, randn

pytestmark = pytest.mark.gpu

ULP = {torch.bfloat16: 2.0**-8, torch.float16: 2.0**-11}


def _rel(a, b, floor):
    a, b = a.double(), b.double()
    return float((a - b).norm() / b.norm().clamp_min(floor))


def _compare(b, lq, lkv, hq, hkv, d, dv, dtype, mask=None, bias=None, dense=None, dropout=0.0, grad_scale=1.0, poison=False):
    """Gradients by the default route against the CUDA-core kernels on the same residuals."""
    dvc = dev()
    q, k, v = randn((b, lq, hq, d), dtype, 1).to(dvc), randn((b, lkv, hkv, d), dtype, 2).to(dvc), randn((b, lkv, hkv, dv), dtype, 3).to(dvc)
    g = (randn((b, lq, hq, dv), torch.float32, 4) * grad_scale).to(dtype).to(dvc)
    lm, residual = M.split_mask(mask, b, lq, lkv)
    assert residual is None
    lb = M.lower_bias_structured(bias, b, hq, lq, lkv)
    mods = A.ScoreMods(lm, lb, dvc, dropout, 1234)
    kvl = None if lm.kv_lengths is None else torch.as_tensor(lm.kv_lengths).to(dvc, torch.int32)
    if poison and kvl is not None:  # keys past the valid length may hold anything
        for i in range(b):
            k[i, int(kvl[i]):] = float("nan")
            v[i, int(kvl[i]):] = float("nan")
    kw = dict(band=lm.band, kv_lengths=kvl, bias=dense, sm_scale=1 / math.sqrt(d),
              mods=mods)
    o, lse = A.attention_forward(q, k, v, return_lse=True, **kw)
    want = A.attention_backward(q, k, v, o, lse, g, impl="b200:generic", bias_grad=dense is not None, **kw)
    got = A.attention_backward(q, k, v, o, lse, g, bias_grad=dense is not None, **kw)
    again = A.attention_backward(q, k, v, o, lse, g, bias_grad=dense is not None, **kw)
    A.check_status(dvc)
    # A row that sees one key has P = 1 and dS = dP - delta = 0: what is computed there is the fp32 noise of two sums of
    # dv products (2^-24 sqrt(dv) |dP| <= 1e-6 of |dO||V|).  Norms are therefore measured against at least 2^-8 of the
    # norm of dv, which makes that noise a 1e-4th of the bound in bf16 and a tenth of it in fp16.
    floor = 2.0**-8 * float(want[2].double().norm())
    for name, x, w, y in zip(("dq", "dk", "dv", "dbias"), got, want, again):
        assert torch.isfinite(x).all(), name
        err = _rel(x, w, 1e-30 if name == "dbias" else floor)
        assert err <= (1e-4 if name == "dbias" else ULP[dtype]), f"{name}: relative difference {err:.2e}"
        assert torch.equal(x, y), f"{name} is not bit-repeatable"
    return got


def _segments(b, n, parts, seed=0):
    g = torch.Generator().manual_seed(seed)
    return torch.sort(torch.randint(0, parts, (b, n), generator=g), dim=1).values.to(torch.int32)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("lq,lkv", [(1, 1), (95, 97), (128, 192), (193, 129), (300, 515)])
def test_latent_head_shape(lq, lkv, dtype):
    """(192, 128): query tiles of 96 rows in the dK/dV kernel, one V stage in the dQ kernel."""
    lens = torch.tensor([lkv, max(1, lkv // 3)], dtype=torch.int32)
    _compare(2, lq, lkv, 4, 4, 192, 128, dtype)
    _compare(2, lq, lkv, 4, 2, 192, 128, dtype, mask=M.CausalMask() & M.KVLenMask(lens), poison=True)
    _compare(2, lq, lkv, 4, 4, 192, 128, dtype, bias=M.CausalAlibiBias(), mask=M.LocalWindowMask(50, 20))


_MODS = {
    "alibi": lambda b, lq, lkv, h: dict(bias=M.CausalAlibiBias(), mask=M.CausalMask()),
    "symmetric_alibi": lambda b, lq, lkv, h: dict(bias=M.SymmetricAlibiBias()),
    "t5": lambda b, lq, lkv, h: dict(bias=M.T5RelativePositionBias(randn((h, 16), torch.float32, 9), num_buckets=16, max_distance=64)),
    "cap_and_scale": lambda b, lq, lkv, h: dict(bias=M.SumBias(M.SoftCappingBias(2.0), M.PerHeadScaleBias(torch.rand(h) + 0.5))),
    "dropout": lambda b, lq, lkv, h: dict(dropout=0.3, mask=M.KVLenMask(torch.tensor([lkv, (lkv + 1) // 2], dtype=torch.int32)), poison=True),
    "heavy_dropout": lambda b, lq, lkv, h: dict(dropout=0.95),
    "prefix": lambda b, lq, lkv, h: dict(mask=M.PrefixLMMask(torch.tensor([min(lkv, 140), 3]))),
    "row_limit": lambda b, lq, lkv, h: dict(mask=M.KeyPaddingMask(torch.arange(1, lq + 1).clamp(max=lkv))),
}


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("name", list(_MODS))
def test_score_modifiers(name, d, dtype):
    for lq, lkv in ((130, 257), (1, 64), (300, 300)):
        _compare(2, lq, lkv, 4, 2, d, d, dtype, **_MODS[name](2, lq, lkv, 4))


@pytest.mark.parametrize("n", [128, 200, 700])
@pytest.mark.parametrize("kind", ["packed", "packed_causal", "reversed_keys", "shuffled", "shared_ids", "prefix"])
def test_segment_masks(kind, n):
    """Segment ranges cut the tile loops of both kernels; ids in any order, per sequence or shared by the batch."""
    seg = _segments(2, n, 6)
    if kind == "reversed_keys":
        mask = M.SameSegmentMask(seg, seg.flip(1))
    elif kind == "shuffled":
        mask = M.SameSegmentMask(seg[:, torch.randperm(n, generator=torch.Generator().manual_seed(3))])
    elif kind == "shared_ids":
        mask = M.BlockDiagonalCausalMask(_segments(1, n, 5))
    elif kind == "prefix":
        mask = M.SameSegmentMask(seg) & M.PrefixLMMask(torch.tensor([n // 2, 5]))
    else:
        mask = (M.BlockDiagonalCausalMask if kind == "packed_causal" else M.BlockDiagonalMask)(seg)
    _compare(2, n, n, 4, 2, 128, 128, torch.bfloat16, mask=mask, bias=M.CausalAlibiBias())
    _compare(2, n, n, 4, 2, 64, 64, torch.float16, mask=mask)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("shape", [(1, 4), (2, 1), (2, 4), (1, 1)])
def test_dense_bias_and_its_gradient(shape, d, dtype):
    for lq, lkv in ((128, 128), (129, 255), (37, 300)):
        dense = randn((*shape, lq, lkv), torch.float32, 7).to(dev())
        lens = torch.tensor([lkv, lkv // 2], dtype=torch.int32)
        _compare(2, lq, lkv, 4, 2, d, d, dtype, mask=M.KVLenMask(lens), dense=dense, poison=True)
        _compare(2, lq, lkv, 4, 2, d, d, dtype, mask=M.CausalMask(), bias=M.CausalAlibiBias(), dense=dense, dropout=0.1)


@pytest.mark.parametrize("fill", [-math.inf, torch.finfo(torch.float32).min, -1e9])
def test_dense_bias_used_as_a_mask(fill):
    """Entries of the type's lowest value, among them whole rows of it: no inf - inf."""
    lq, lkv = 140, 260
    dense = randn((1, 4, lq, lkv), torch.float32, 7)
    dense[:, :, :, 150:] = fill
    if fill != -math.inf:  # (a row of -inf has no defined softmax)
        dense[:, :, 17] = fill
    _compare(2, lq, lkv, 4, 4, 64, 64, torch.bfloat16, dense=dense.to(dev()))


def test_fp16_gradients_far_from_one():
    """fp16 packs P and dS scaled: output gradients of 1e-3 and of 100 keep what fp32 arithmetic gave."""
    for scale in (1e-3, 1.0, 100.0):
        _compare(2, 200, 300, 4, 2, 64, 64, torch.float16, bias=M.SymmetricAlibiBias(), grad_scale=scale)
