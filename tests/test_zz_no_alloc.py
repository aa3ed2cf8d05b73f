"""The allocation-free decode entry point, called through the C ABI.

Some callers can hand the library nothing but their inputs and outputs: inside a
compiler-planned custom call every buffer is fixed ahead of time and cudaMalloc is
off limits, and the same holds while a device allocator is locked or out of
memory.  ``pjx_attn_decode_splitkv_static`` keeps its per-split partials in a
fixed array inside the library for them.  This file checks it against the
workspace-taking entry point on two calls in a row (the second with other inputs,
shorter sequences and a different split length, so that leftovers of the first
call sit in the shared array), and that oversized calls are refused.

It is collected last on purpose: a run that stops at the first failure has then
already run every other test.
"""

import ctypes as C
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


def _ptr(t):
    return None if t is None else C.c_void_p(t.data_ptr())


def _static_call(L, q, k, v, lens, sc, split_len, o_s, lse_s):
    from probjax_b200 import _lib
    from probjax_b200.attention import _DTYPES

    B, Lq, Hq, D = q.shape
    cap, Hkv, Dv = k.shape[1], k.shape[2], v.shape[3]
    stream = C.c_void_p(torch.cuda.current_stream(q.device).cuda_stream)
    rc = L.pjx_attn_decode_splitkv_static(_ptr(q), _ptr(k), _ptr(v), _ptr(lens), _ptr(o_s), _ptr(lse_s),
                                          B, Lq, Hq, Hkv, D, Dv, cap, _DTYPES[q.dtype], sc, split_len, stream)
    _lib.check(rc)


def _call_pair(L, q, k, v, lens, sc, split_len):
    """(static entry point, workspace entry point) results for the same inputs.  Every tensor is
    allocated before the static call, and the device's free memory and torch's allocation count
    are read on both sides of it: the entry point itself must not allocate."""
    from probjax_b200 import _lib
    from probjax_b200.attention import _DTYPES

    dev = q.device
    B, Lq, Hq, D = q.shape
    cap, Hkv, Dv = k.shape[1], k.shape[2], v.shape[3]
    stream = C.c_void_p(torch.cuda.current_stream(dev).cuda_stream)
    o_s = torch.empty(B, Lq, Hq, Dv, dtype=q.dtype, device=dev)
    lse_s = torch.empty(B, Hq, Lq, dtype=torch.float32, device=dev)
    o_w = torch.empty_like(o_s)
    lse_w = torch.empty_like(lse_s)
    need = L.pjx_attn_decode_workspace_bytes(B, Lq, Hq, Hkv, Dv, cap, split_len)
    ws = torch.empty(need, dtype=torch.uint8, device=dev)
    _static_call(L, q, k, v, lens, sc, split_len, o_s, lse_s)  # first use: module load, address look-up
    torch.cuda.synchronize(dev)
    o_s.zero_()
    free0, held0 = torch.cuda.mem_get_info(dev)[0], torch.cuda.memory_allocated(dev)
    _static_call(L, q, k, v, lens, sc, split_len, o_s, lse_s)
    torch.cuda.synchronize(dev)
    free1, held1 = torch.cuda.mem_get_info(dev)[0], torch.cuda.memory_allocated(dev)
    assert held1 == held0, "the allocation-free entry point went through torch's allocator"
    assert free1 >= free0, f"device free memory fell by {free0 - free1} bytes across the allocation-free call"
    rc = L.pjx_attn_decode_splitkv(_ptr(q), _ptr(k), _ptr(v), _ptr(lens), _ptr(o_w), _ptr(lse_w),
                                   B, Lq, Hq, Hkv, D, Dv, cap, _DTYPES[q.dtype], sc, split_len, 0, _ptr(ws), need, stream)
    _lib.check(rc)
    torch.cuda.synchronize(dev)
    return (o_s, lse_s), (o_w, lse_w)


def test_static_scratch_decode_matches_workspace_decode_twice():
    import oracle
    from probjax_b200 import _lib

    L = _lib.lib()
    dev = torch.device("cuda", 0)
    assert L.pjx_attn_decode_static_scratch_bytes() == 16 * 1024 * 1024
    g = torch.Generator().manual_seed(123)
    # (dtype, B, Lq, Hq, Hkv, D, capacity, lengths, split_len); the later calls are shorter or of another
    # shape, so leftovers of the earlier ones sit in the shared array
    calls = [
        (torch.bfloat16, 4, 1, 32, 8, 128, 4096, [4096, 1000, 2500, 77], 256),
        (torch.bfloat16, 4, 1, 32, 8, 128, 4096, [300, 4096, 1, 0], 0),
        (torch.float16, 3, 2, 8, 2, 64, 1536, [1536, 65, 700], 128),  # fp16, D = 64, two query rows, GQA
    ]
    for dtype, B, Lq, Hq, Hkv, D, cap, lens, split_len in calls:
        sc = 1 / math.sqrt(D)
        lens = torch.tensor(lens, dtype=torch.int32)
        q = torch.randn(B, Lq, Hq, D, generator=g).to(dtype)
        k = torch.randn(B, cap, Hkv, D, generator=g).to(dtype)
        v = torch.randn(B, cap, Hkv, D, generator=g).to(dtype)
        (o_s, lse_s), (o_w, lse_w) = _call_pair(L, q.to(dev), k.to(dev), v.to(dev), lens.to(dev), sc, split_len)
        # same kernels, same split geometry, same arithmetic: bit-identical to the workspace entry point
        assert torch.equal(o_s, o_w)
        assert torch.equal(lse_s, lse_w)
        # and within the parity bounds of the fp32 oracle: 16-bit outputs 2e-2, LSE 1e-3
        want, want_lse = oracle.xla_attention(q, k, v, kv_lengths=lens, sm_scale=sc, return_lse=True)
        assert float((o_s.float().cpu() - want.float()).abs().max()) <= 2e-2
        fin = torch.isfinite(want_lse)
        assert torch.equal(torch.isinf(lse_s.cpu()), ~fin)
        assert float((lse_s.cpu()[fin] - want_lse[fin]).abs().max()) <= 1e-3
        assert (o_s[lens.to(dev) == 0] == 0).all()


def test_static_scratch_decode_rejects_what_it_cannot_hold():
    from probjax_b200 import _lib

    L = _lib.lib()
    dev = torch.device("cuda", 0)
    B, Hq, Hkv, D, cap = 64, 32, 8, 128, 32768
    q = torch.zeros(B, 1, Hq, D, dtype=torch.bfloat16, device=dev)
    o = torch.empty_like(q)
    stream = C.c_void_p(torch.cuda.current_stream(dev).cuda_stream)
    # 64 x 8 x 512 splits x 4 rows x 129 floats is far beyond 16 MiB; the caches are never touched
    rc = L.pjx_attn_decode_splitkv_static(_ptr(q), _ptr(q), _ptr(q), None, _ptr(o), None,
                                          B, 1, Hq, Hkv, D, D, cap, _lib.PJX_BF16, 0.1, 64, stream)
    assert rc == _lib.PJX_ERR_WORKSPACE and "split_len" in _lib.last_error()
    # fp32 is not a streaming-kernel case
    rc = L.pjx_attn_decode_splitkv_static(_ptr(q), _ptr(q), _ptr(q), None, _ptr(o), None,
                                          1, 1, Hq, Hkv, D, D, 64, _lib.PJX_F32, 0.1, 64, stream)
    assert rc == _lib.PJX_ERR_UNSUPPORTED


def _pool_high_water(dev, reset=False):
    """Most bytes the device's stream-ordered pool had in use at a time (since the last reset)."""
    rt = C.CDLL("libcudart.so.12")
    pool, value = C.c_void_p(), C.c_uint64(0)
    assert rt.cudaDeviceGetDefaultMemPool(C.byref(pool), dev.index) == 0
    if reset:
        assert rt.cudaMemPoolSetAttribute(pool, 8, C.byref(value)) == 0  # cudaMemPoolAttrUsedMemHigh
    assert rt.cudaMemPoolGetAttribute(pool, 8, C.byref(value)) == 0
    return value.value


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("kind", ["segments", "latent"])
def test_backward_keeps_its_scratch_in_the_workspace(kind, dtype):
    """With the sized workspace the call takes nothing from the stream-ordered pool.  With the one of the row vectors alone
    it is still accepted: bf16 visits every tile (those that cannot match add exact zeros), fp16 runs on the CUDA cores."""
    from _gpu_util import dev, randn
    from probjax_b200 import _lib
    from probjax_b200 import attention as A
    from probjax_b200 import masks as M

    b, l, h, d, dv = 2, 300, 4, *((192, 128) if kind == "latent" else (128, 128))
    dvc, L = dev(), _lib.lib()
    q, k, v, g = (randn((b, l, h, n), dtype, i).to(dvc) for i, n in enumerate((d, d, dv, dv)))
    mods = None
    if kind == "segments":
        ids = torch.repeat_interleave(torch.arange(3, dtype=torch.int32), torch.tensor([140, 100, 60]))[None].repeat(b, 1)
        mods = A.ScoreMods(M.split_mask(M.SameSegmentMask(ids), b, l, l)[0], M.lower_bias_structured(None, b, h, l, l), dvc, 0.0, 0)
    kw = dict(sm_scale=1 / math.sqrt(d), mods=mods)
    o, lse = A.attention_forward(q, k, v, return_lse=True, **kw)
    want = A.attention_backward(q, k, v, o, lse, g, **kw)
    slow = A.attention_backward(q, k, v, o, lse, g, impl="b200:generic", **kw)
    torch.cuda.synchronize(dvc)
    held = _pool_high_water(dvc, reset=True)
    again = A.attention_backward(q, k, v, o, lse, g, **kw)
    torch.cuda.synchronize(dvc)
    assert _pool_high_water(dvc) == held
    assert all(torch.equal(x, y) for x, y in zip(again, want))

    code = A._DTYPES[dtype]
    need = L.pjx_attn_bwd_workspace_bytes(b, l, h)
    assert need < L.pjx_attn_bwd_mod_workspace_bytes(b, l, l, h, h, code)
    ws = torch.empty(need, dtype=torch.uint8, device=dvc)
    got = [torch.empty_like(t) for t in (q, k, v)]
    rc = L.pjx_attn_bwd_mod(*(A._ptr(t) for t in (q, k, v, o, lse, g, *got)), None, None, 0, 0, None, b, l, l, h, h, d, dv, code,
                            -(1 << 30), 1 << 30, kw["sm_scale"], A.ScoreMods.arg(mods), 0, A._ptr(ws), need,
                            A._ptr(A._status_word(dvc)), A._stream(dvc))
    _lib.check(rc)
    A.check_status(dvc)
    assert all(torch.equal(x, y) for x, y in zip(got, want if dtype == torch.bfloat16 else slow))
