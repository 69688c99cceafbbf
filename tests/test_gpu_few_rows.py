"""The kernels of a decode step's few rows at the edges of their forms: the map a CTA a row, the spread expansion, the folded scan."""

import numpy as np
import pytest
import torch

from helpers import cuda

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,heads,group,dh,off,used,d_idx,dtype", [
    (1, 40, 5, 128, 0, 128, 64, torch.bfloat16), (128, 8, 4, 128, 32, 96, 32, torch.bfloat16), (33, 3, 1, 72, 8, 61, 128, torch.float32),
    (7, 64, 1, 576, 0, 576, 64, torch.bfloat16), (129, 8, 2, 128, 0, 128, 64, torch.bfloat16)])
def test_the_map_of_a_few_rows(rows, heads, group, dh, off, used, d_idx, dtype):
    """Unit rows against 64 bits: an fp32 sum of n terms is off by some n^0.5 2^-24 of its size, 2e-5 at 36,864 terms."""
    from lsa_b200 import ops

    gen = torch.Generator(device="cuda").manual_seed(rows)
    x = torch.randn(rows, heads, dh, device="cuda", generator=gen).to(dtype)
    w = torch.randn(heads // group * used, d_idx, device="cuda", generator=gen).bfloat16()
    summed = x[..., off:off + used].double().view(rows, heads // group, group, used).sum(2).reshape(rows, -1)
    want = torch.nn.functional.normalize(summed @ w.double(), dim=-1)
    got, half = ops.index_map(x, w, group=group, dh_off=off, dh_used=used, also_bf16=True)
    assert (got.double() - want).abs().max() <= 2e-5 and torch.equal(half, got.bfloat16())
    plain = ops.index_map(x, w, group=group, dh_off=off, dh_used=used, normalize=False)
    assert (plain.double() - summed @ w.double()).abs().max() <= 2e-5 * (summed @ w.double()).norm(dim=-1).max()


@pytest.mark.parametrize("rows,heads,d_in,d_out", [(1, 64, 576, 2048), (8, 64, 576, 40), (3, 2, 8, 9), (2, 20, 2048, 64)])
def test_heads_summed_in_shared_memory_are_the_heads_summed(rows, heads, d_in, d_out):
    """Rows whose heads are staged against the same rows at a stride that is not: bit for bit (the sums keep the heads' order)."""
    from lsa_b200 import ops

    gen = torch.Generator(device="cuda").manual_seed(d_in)
    x = torch.randn(rows, heads, d_in, device="cuda", generator=gen).bfloat16()
    w = torch.randn(d_out, d_in, device="cuda", generator=gen).bfloat16()
    apart = torch.zeros(rows, heads, d_in + 2, device="cuda", dtype=torch.bfloat16)[..., :d_in].copy_(x)
    assert apart.stride(1) % 8
    assert torch.equal(ops.rows_linear(x, w, sum_heads=True), ops.rows_linear(apart, w, sum_heads=True))
