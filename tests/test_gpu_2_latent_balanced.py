"""Latent decode with the split length chosen on the device from the valid lengths, against explicit splits.

Both compute every row in fp32 and round it once; the order of the combination differs, so an element may differ by
one unit in the last place (2^-8 in bf16, 2^-11 in fp16 of it, hence of the norm) and the log-sum-exp by fp32 rounding.
"""

import pytest
import torch

import probjax_b200 as pj
from _gpu_util import dev, randn

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("lens,cap,heads,r", [
    ([5000], 5000, 16, 576),                                  # one sequence
    ([0, 1, 127, 128, 129, 4096], 4096, 16, 512),             # an empty one, edges of a block of 128 keys
    ([8192, 3, 3, 3], 8192, 32, 576),                         # one long among short, two row groups
    ([16384, 16384, 9000, 700, 2048, 1, 15000, 8000], 16384, 16, 576),  # the tcgen05 kernel
    ([(37 * i) % 900 + 1 for i in range(33)], 1024, 16, 576),  # more sequences than lanes of a warp
    ([0, 0], 600, 16, 512),
])
def test_against_explicit_splits(lens, cap, heads, r, dtype):
    d = dev()
    b = len(lens)
    q, cache = randn((b, 1, heads, r), dtype, 1).to(d), randn((b, cap, r), dtype, 2).to(d)
    lt = torch.tensor(lens, dtype=torch.int32, device=d)
    for i, n in enumerate(lens):
        cache[i, n:] = float("nan")  # a cache tail that was never written
    got, lse = pj.mla_decode(q, cache, kv_lengths=lt, sm_scale=0.05, return_lse=True)
    want, want_lse = pj.mla_decode(q, cache, kv_lengths=lt, sm_scale=0.05, split_len=256, return_lse=True)
    again = pj.mla_decode(q, cache, kv_lengths=lt, sm_scale=0.05)
    pj.check_status(d)
    assert torch.isfinite(got).all() and torch.equal(got, again)
    tol = {torch.bfloat16: 2.0**-8, torch.float16: 2.0**-11}[dtype]
    assert float((got.double() - want.double()).norm()) <= tol * float(want.double().norm())
    empty = torch.tensor([n == 0 for n in lens], device=d)
    assert (got[empty] == 0).all() and torch.isinf(lse[empty]).all()
    assert float((lse[~empty] - want_lse[~empty]).abs().max() if (~empty).any() else 0.0) <= 1e-4
