"""Tensor-core backward of the calls that carry score modifiers, a dense bias or the latent head shape.

Its P and dS enter the products as 16 + 16 bits, so its 16-bit gradients may differ from those of the exact-fp32
CUDA-core kernels (same inputs, same saved o and lse) by the rounding of the result only: one unit in the last
place of an element, 2^-8 (bf16) or 2^-11 (fp16) of it, hence at most that of the norm.  The bias gradient is fp32;
its error is that of the scores and of dP, sums of D products (2^-24 sqrt(D) each, doubled for the unit's
truncation), times the cancellation in dP - delta: 1e-4 of the norm leaves a factor of ten.  That bound is one unit of the
whole norm and does not show whether the low halves are there: the comparisons with float64 further down do, row by row.
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


def test_large_grids():
    """More CTAs than SMs in both kernels, 19 tiles along both axes, a last tile of 5 rows."""
    n = 18 * 128 + 5
    _compare(1, n, n, 16, 4, 128, 128, torch.bfloat16, mask=M.BlockDiagonalCausalMask(_segments(1, n, 5)), bias=M.CausalAlibiBias())
    _compare(2, n, n, 8, 8, 192, 128, torch.float16, mask=M.CausalMask())
    _compare(3, n, 1025, 8, 8, 64, 64, torch.float16, dense=randn((1, 8, n, 1025), torch.float32, 7).to(dev()))


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


# ------------------------------------------------------------------------------------------- against float64


def _float64_backward(q, k, v, o, lse, g, keep, sm_scale, bias=None):
    """Gradients in float64 from the residuals the kernels get, ``keep [B, 1|H, Lq, Lkv]``, and for each of dq, dk, dv
    what fp32 arithmetic may add to it: 2^-20 (sums of D <= 192 products, the exponential, and sums over the keys, a
    dozen roundings of 2^-24) of the sum of the magnitudes of its terms, P |dP| and P |delta| before they cancel."""
    G = q.shape[2] // k.shape[2]
    qd, od, gd = (t.double().transpose(1, 2) for t in (q, o, g))
    kd, vd = (t.double().transpose(1, 2).repeat_interleave(G, 1) for t in (k, v))
    s = qd @ kd.transpose(2, 3) * sm_scale
    if bias is not None:
        s = s + bias.double()
    p = torch.where(keep, torch.exp(s - lse.double()[..., None]), 0.0)
    dp, delta = gd @ vd.transpose(2, 3), (od * gd).sum(3, keepdim=True)
    ds, mag = p * (dp - delta), p * (dp.abs() + delta.abs())

    def per_key_head(x):
        return x.unflatten(1, (-1, G)).sum(2).transpose(1, 2)

    want = [(ds @ kd * sm_scale).transpose(1, 2), per_key_head(ds.transpose(2, 3) @ qd * sm_scale), per_key_head(p.transpose(2, 3) @ gd)]
    noise = [(mag @ kd.abs() * sm_scale).transpose(1, 2), per_key_head(mag.transpose(2, 3) @ qd.abs() * sm_scale),
             per_key_head(p.transpose(2, 3) @ gd.abs())]
    return want, [2.0**-20 * n for n in noise]


def _segment_ids(lengths):
    return torch.repeat_interleave(torch.arange(len(lengths), dtype=torch.int32), torch.tensor(lengths))[None].repeat(2, 1)


@pytest.mark.parametrize("d,dv", [(64, 64), (128, 128), (192, 128)])
@pytest.mark.parametrize("spread", [1e3, 1e6])
@pytest.mark.parametrize("where", ["row", "head", "sequence", "value", "uniform"])
def test_fp16_rows_keep_their_bits_beside_much_larger_ones(where, spread, d, dv):
    """fp16 has no range to spare for the low parts: a row of dO (of one head, of one sequence), or of V, far above the
    rest must not take bits from the others.  Every row of every gradient is held to its own magnitude: the rounding
    to fp16 (2^-11 of an element, 2^-25 below the normal range) and the fp32 term of ``_float64_backward``."""
    b, l, hq, hkv = 2, 200, 4, 2
    dvc, dtype = dev(), torch.float16
    q, k, v = randn((b, l, hq, d), dtype, 1), randn((b, l, hkv, d), dtype, 2), randn((b, l, hkv, dv), dtype, 3)
    g = randn((b, l, hq, dv), torch.float32, 4)
    low = min(1.0, 5e4 / (4 * spread))  # the large entries stay finite in fp16
    if where == "value":  # 5e3 above the rest at most, in a document of its own: P dP of the others does not feel it
        v[0, 150, 1] *= min(spread, 5e3)
    elif where == "uniform":
        g = g * low
    else:
        big = torch.zeros(b, l, hq, 1)
        big[{"row": (0, 7, 1), "head": (slice(None), slice(None), 2), "sequence": (1,)}[where]] = 1.0
        g = g * torch.where(big > 0, low * spread, low)
    q, k, v, g = (t.to(dvc) for t in (q, k, v, g.clamp(-6e4, 6e4).to(dtype)))
    mask = M.BlockDiagonalMask(_segment_ids([60, 71, 69]))
    mods = A.ScoreMods(M.split_mask(mask, b, l, l)[0], M.lower_bias_structured(None, b, hq, l, l), dvc, 0.0, 0)
    kw = dict(sm_scale=1 / math.sqrt(d), mods=mods)
    o, lse = A.attention_forward(q, k, v, return_lse=True, **kw)
    got = A.attention_backward(q, k, v, o, lse, g, **kw)
    A.check_status(dvc)
    keep = mask.dense(l, l, batch_size=b, num_heads=1).to(dvc).reshape(b, 1, l, l)
    want, noise = _float64_backward(q, k, v, o, lse, g, keep, kw["sm_scale"])
    for name, x, w, n in zip(("dq", "dk", "dv"), got, want, noise):
        fits = w.abs() < 6.5e4
        bound = (2.0**-11 * w.abs() + 2.0**-25 + n).norm(dim=3)
        err = torch.where(fits, x.double() - w, 0.0).norm(dim=3)
        worst = float((err / bound).max())
        assert worst <= 1.0, f"{name}: a row is off by {worst:.3g} of its bound"


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("kind", ["latent", "packed", "dense", "dense_128"])
def test_only_the_rounding_of_the_result_is_left(kind, dtype):
    """Against float64 the error is that of rounding the result to 16 bits, as with fp32 arithmetic throughout.  P and dS
    without their low parts add 2^-9 (bf16) or 2^-12 (fp16) of each term and raise it by half."""
    b, l, hq = 2, 515, 4
    d, dv = {"latent": (192, 128), "packed": (128, 128), "dense": (64, 64), "dense_128": (128, 128)}[kind]
    dvc = dev()
    q, k, v = randn((b, l, hq, d), dtype, 1).to(dvc), randn((b, l, 2, d), dtype, 2).to(dvc), randn((b, l, 2, dv), dtype, 3).to(dvc)
    g = randn((b, l, hq, dv), dtype, 4).to(dvc)
    keep, dense, kw = torch.ones(b, 1, l, l, dtype=torch.bool, device=dvc), None, dict(sm_scale=1 / math.sqrt(d))
    if kind == "packed":
        mask = M.BlockDiagonalMask(_segment_ids([200, 115, 200]))
        keep = mask.dense(l, l, batch_size=b, num_heads=1).to(dvc).reshape(b, 1, l, l)
        kw["mods"] = A.ScoreMods(M.split_mask(mask, b, l, l)[0], M.lower_bias_structured(None, b, hq, l, l), dvc, 0.0, 0)
    elif kind != "latent":
        dense = kw["bias"] = randn((1, hq, l, l), torch.float32, 7).to(dvc)
    o, lse = A.attention_forward(q, k, v, return_lse=True, **kw)
    got = A.attention_backward(q, k, v, o, lse, g, **kw)
    A.check_status(dvc)
    want, noise = _float64_backward(q, k, v, o, lse, g, keep, kw["sm_scale"], dense)
    for name, x, w, n in zip(("dq", "dk", "dv"), got, want, noise):
        rounding = float((w.to(dtype).double() - w).norm())
        err = float((x.double() - w).norm())
        assert err <= 1.001 * rounding + float(n.norm()), f"{name}: {err / rounding:.5f} of the rounding error"


# ------------------------------------------------------------------------------------------- many short sequences


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("b,lq,lkv,hq,hkv,planes,d", [
    (8, 64, 64, 4, 4, (1, 1), 64),      # one tile, 32 pairs: a cluster of eight
    (33, 40, 72, 2, 2, (1, 1), 128),    # one tile, 66 pairs: sixteen CTAs, slices of unequal length
    (64, 130, 33, 2, 1, (1, 2), 64),    # four tiles, an odd number of keys, 64 pairs each
    (2, 260, 200, 16, 4, (2, 1), 64),   # three by two tiles per sequence, 16 heads each: clusters of four
])
def test_bias_gradient_shared_by_many_pairs(b, lq, lkv, hq, hkv, planes, d, dtype):
    """A bias that many (sequence, head) pairs share: its gradient is summed by clusters of CTAs, among them slices of pairs
    whose keys are all past the valid length.  The order of the sum differs from the oracle route's by the pairs: 2^-24
    sqrt(pairs) of the magnitudes, far inside ``_compare``'s bound."""
    dense = randn((*planes, lq, lkv), torch.float32, 7).to(dev())
    lens = torch.tensor([(i * 29) % (lkv + 1) for i in range(b)], dtype=torch.int32)
    _compare(b, lq, lkv, hq, hkv, d, d, dtype, mask=M.KVLenMask(lens), dense=dense, poison=True)
    _compare(b, lq, lkv, hq, hkv, d, d, dtype, mask=M.LocalWindowMask(20, 9), bias=M.CausalAlibiBias(), dense=dense)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("n", [1, 16, 32, 33])
@pytest.mark.parametrize("planes", [(1, 1), (1, 4), (40, 1), None])
def test_one_tile_calls(planes, n, dtype):
    """Up to 32 queries and keys and more pairs than SMs run on the CUDA cores, a shared bias summed over the pairs from the
    workspace in a fixed order; 33 is the first size past the rule."""
    # (two keys or more, or none: a row that sees one key has dS = dP - delta = 0, and a bias gradient of nothing else is noise)
    lens = torch.tensor([(i * 7) % 31 + 2 if i % 8 else 0 for i in range(40)], dtype=torch.int32)
    dense = None if planes is None else randn((*planes, n, 32), torch.float32, 7).to(dev())
    for hkv in (4, 2):  # (2: below a wave of key heads, on the tensor cores)
        _compare(40, n, 32, 4, hkv, 64, 64, dtype, mask=M.KVLenMask(lens), dense=dense, bias=M.SymmetricAlibiBias(), poison=True)


def _time_us(fn):
    start, end = (torch.cuda.Event(enable_timing=True) for _ in range(2))
    best = math.inf
    for _ in range(6):
        torch.cuda._sleep(1_000_000)
        start.record()
        for _ in range(5):
            fn()
        end.record()
        end.synchronize()
        best = min(best, start.elapsed_time(end) * 200)
    return best


@pytest.mark.parametrize("alibi", [False, True])
@pytest.mark.parametrize("b,n,h,planes,bias_grad", [(64, 64, 16, 1, False), (64, 64, 16, 1, True), (256, 16, 8, 1, True), (256, 16, 8, 8, False)])
def test_many_short_sequences_are_not_slower_than_on_cuda_cores(b, n, h, planes, bias_grad, alibi):
    """Short sequences that share a bias: the default route takes at most 1.3 times as long as the CUDA-core kernels (every SM
    reading the last line of the bias: 1.4 times; one CTA walking all pairs of a tile: 5.4 times; tcgen05 tiles filled to a
    sixteenth: 3.2 times)."""
    dvc = dev()
    q, k, v, g = (randn((b, n, h, 64), torch.bfloat16, i).to(dvc) for i in range(4))
    kw = dict(sm_scale=0.125, bias=randn((1, planes, n, n), torch.float32, 5).to(dvc))
    if alibi:
        kw["mods"] = A.ScoreMods(M.split_mask(None, b, n, n)[0], M.lower_bias_structured(M.CausalAlibiBias(), b, h, n, n), dvc, 0.0, 0)
    o, lse = A.attention_forward(q, k, v, return_lse=True, **kw)
    kw["bias_grad"] = bias_grad
    got = _time_us(lambda: A.attention_backward(q, k, v, o, lse, g, **kw))
    base = _time_us(lambda: A.attention_backward(q, k, v, o, lse, g, impl="b200:generic", **kw))
    assert got <= 1.3 * base, f"{got:.1f} us against {base:.1f}"


@pytest.mark.parametrize("b,n", [(32, 64), (40, 16)])
def test_shared_bias_gradient_under_capture(b, n):
    """The cluster launch and the sum over pairs replay from a graph, on new inputs in the captured buffers."""
    dvc = dev()
    q, k, v, g = (randn((b, n, 4, 64), torch.bfloat16, i).to(dvc) for i in range(4))
    kw = dict(sm_scale=0.125, bias=randn((1, 1, n, n), torch.float32, 5).to(dvc))

    def step():
        o, lse = A.attention_forward(q, k, v, return_lse=True, **kw)
        return A.attention_backward(q, k, v, o, lse, g, bias_grad=True, **kw)

    side = torch.cuda.Stream(dvc)
    with torch.cuda.stream(side):
        step()
    side.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=side):
        got = step()
    for t in (q, k, v, g):
        t.copy_(t.flip(0) * 0.5)
    graph.replay()
    torch.cuda.synchronize(dvc)
    assert all(torch.equal(x, y) for x, y in zip(got, step()))
