"""The dense reads on the tensor cores (causal, banded, masked by lists) and the lists as bits, at the edges of their tiles."""

import numpy as np
import pytest
import torch

from helpers import cuda, layer_inputs

pytestmark = pytest.mark.gpu


def _read(q, k, v, keep):
    """Attention in 64 bits over the keys `keep` [R, n] names: (out [R, Hq, dh], lse [R, Hq]); rows that read nothing are zero."""
    group = q.shape[1] // k.shape[1]
    scores = torch.einsum("qhd,khd->hqk", q.double(), k.double().repeat_interleave(group, dim=1)) * q.shape[2] ** -0.5
    scores.masked_fill_(~keep, -float("inf"))
    lse = scores.logsumexp(-1)
    weights = (scores - lse.clamp_min(-1e30)[..., None]).exp()
    return torch.einsum("hqk,khd->qhd", weights, v.double().repeat_interleave(group, dim=1)), lse.t()


@pytest.mark.parametrize("R,first,window,sink", [(128, 0, 1, 0), (200, 1000, 1, 4), (129, 255, 128, 64), (300, 0, 129, 4),
                                                 (513, 385, 256, 1), (256, 3, 4000, 7), (640, 700, 513, 64)])
def test_band_at_the_edges_of_its_tiles(R, first, window, sink):
    """Output and log-sum-exp of a band against 64 bits; two terms leave 2^-17 of a probability and the fp32 sums less: 2^-16 in
    all."""
    from lsa_b200 import ops

    n = first + R
    q, k, v = (cuda(x, torch.bfloat16) for x in layer_inputs(n, 4, 2, 128, 16, n + window))
    pos, key = first + torch.arange(R, device="cuda")[:, None], torch.arange(n, device="cuda")
    keep = (key <= pos) & ((key > pos - window) | (key < sink))
    want, want_lse = _read(q[first:], k, v, keep)
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    out, lse = ops.band_attend(q[first:], k, v, first, window, sink, 128 ** -0.5, status=status)
    assert (out.double() - want).norm() <= 2 ** -16 * want.norm() and int(status) == 0
    assert (lse.double() - want_lse).abs().max() <= 1e-4


def test_a_running_maximum_that_grows_keeps_the_sums():
    """Scores that climb by powers of two from tile to tile, down again, and past what a probability of 2^8 covers."""
    from lsa_b200 import ops

    n = 1024
    gen = torch.Generator(device="cuda").manual_seed(0)
    q, k, v = (torch.randn(n, 2, 128, device="cuda", generator=gen) for _ in range(3))
    climb = torch.tensor([0.1, 3.0, 0.5, 9.0, 27.0, 1.0, 60.0, 2.0], device="cuda").repeat_interleave(128)[:, None, None]
    q, k, v = q.bfloat16(), (0.7 * q * climb + k).bfloat16(), v.bfloat16()
    keep = torch.ones(n, n, device="cuda").tril().bool()
    want, _ = _read(q, k, v, keep)
    got = ops.causal_attend(q, k, v, 0, 128 ** -0.5, out=torch.empty(n, 2, 128, device="cuda"))
    # (scores of up to 600 in log2: an fp32 product is off by 2^-24 of it, 2^-14 of a probability, and rounds in sums of 128)
    assert (got.double() - want).norm() <= 2 ** -12 * want.norm()
