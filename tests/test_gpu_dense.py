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


@pytest.mark.parametrize("listed", [False, True])
def test_a_maximum_that_moves_at_every_tile_scales_whole_rows_of_o(listed):
    """Scores that climb by 9 to 20 in log2 a key tile, so that nearly every product finds an O that two threads a row have just
    scaled: more CTAs than SMs, again and again, against 64 bits and bit for bit against the first time. Exponents of up to 700 in
    fp32 are off by 2^-24 of it and the 128 terms of a product by some bits more: 2^-12 of a probability."""
    from lsa_b200 import ops

    R, n, Hq, Hkv = 1024, 4096, 40, 8
    gen = torch.Generator(device="cuda").manual_seed(int(listed))
    towards = torch.nn.functional.normalize(torch.randn(Hkv, 128, device="cuda", generator=gen), dim=-1)
    tile = torch.arange(n, device="cuda")[:, None, None] // 128
    k = (towards * tile + 0.3 * torch.randn(n, Hkv, 128, device="cuda", generator=gen)).bfloat16()
    steep = torch.empty(R, Hq, 1, device="cuda").uniform_(9.0, 20.0, generator=gen) * 128 ** 0.5 * 0.6931471805599453
    q = (steep * towards.repeat_interleave(Hq // Hkv, dim=0)).bfloat16()
    v = torch.randn(n, Hkv, 128, device="cuda", generator=gen).bfloat16()
    keep = torch.arange(n, device="cuda") <= n - R + torch.arange(R, device="cuda")[:, None]
    if listed:
        keep &= torch.rand(R, n, device="cuda", generator=gen) < 0.5
        mask = _bits(keep)
    out = torch.empty(R, Hq, 128, device="cuda")
    read = lambda: ops.listed_attend(q, k, v, n - R, mask, 128 ** -0.5, out) if listed else \
        ops.causal_attend(q, k, v, n - R, 128 ** -0.5, out=out)
    first = read().clone()
    for h in range(Hkv):
        heads = slice(h * Hq // Hkv, (h + 1) * Hq // Hkv)
        want, _ = _read(q[:, heads], k[:, h:h + 1], v[:, h:h + 1], keep)
        assert (first[:, heads].double() - want).norm() <= 2 ** -12 * want.norm()
    for _ in range(40):
        assert torch.equal(read(), first)


def _bits(keep):
    """keep [R, n] bool as words [tiles, R, 4] int32."""
    R, n = keep.shape
    tiles = -(-n // 128)
    bits = torch.zeros(R, tiles * 128, dtype=torch.int64, device=keep.device)
    bits[:, :n] = keep
    words = (bits.view(R, tiles, 4, 32) << torch.arange(32, device=keep.device)).sum(-1)
    return torch.where(words >= 2 ** 31, words - 2 ** 32, words).to(torch.int32).permute(1, 0, 2).contiguous()


@pytest.mark.parametrize("R,first,Hq,Hkv", [(1, 0, 1, 1), (127, 1, 2, 1), (128, 0, 5, 1), (129, 127, 4, 2), (255, 0, 2, 2),
                                            (256, 640, 8, 1), (257, 129, 3, 3), (640, 77, 6, 2)])
def test_masked_rows_read_the_keys_they_list(R, first, Hq, Hkv):
    """Random lists, rows that list nothing, one key or every key; and a value and a key that are not finite reach the rows that
    list them alone. 2^-16 as above."""
    from lsa_b200 import ops

    n = first + R
    q, k, v = (cuda(x, torch.bfloat16) for x in layer_inputs(n, Hq, Hkv, 128, 16, n))
    q = q[first:]
    gen = torch.Generator(device="cuda").manual_seed(n)
    keep = torch.rand(R, n, device="cuda", generator=gen) < torch.rand(R, 1, device="cuda", generator=gen)
    keep &= torch.arange(n, device="cuda") <= first + torch.arange(R, device="cuda")[:, None]
    keep[0] = False
    if R > 2:
        keep[1] = False
        keep[1, first] = True
        keep[2] = torch.arange(n, device="cuda") <= first + 2
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    read = lambda dtype: ops.listed_attend(q, k, v, first, _bits(keep), 128 ** -0.5,
                                           torch.empty(R, Hq, 128, device="cuda", dtype=dtype), status)
    want, _ = _read(q, k, v, keep)
    got = read(torch.float32)
    assert (got.double() - want).norm() <= 2 ** -16 * want.norm() and not got[0].any()
    assert (read(torch.bfloat16).double() - want).abs().max() <= 2 ** -8 * want.abs().max() and int(status) == 0
    for x, at, what in ((v, first, float("inf")), (k, first, float("nan"))):
        kept = x[at, 0, 5].clone()
        x[at, 0, 5] = what
        odd = ~read(torch.float32).isfinite().all(-1)
        x[at, 0, 5] = kept
        heads = torch.arange(Hq, device="cuda") < Hq // Hkv
        assert torch.equal(odd, keep[:, first, None] & heads)


@pytest.mark.parametrize("share,most", [(1.0, 100), (0.25, 40)])
def test_a_value_that_is_not_finite_costs_a_bounded_time(share, most):
    """An infinity in a value that most rows walk over (all of a KV head's rows are read again): 40 and 12 times the clean read
    here, where a key at a time took 223 and 95."""
    from lsa_b200 import ops

    R, Hq, Hkv = 4096, 16, 2
    gen = torch.Generator(device="cuda").manual_seed(0)
    q, k, v = (torch.randn(R, h, 128, device="cuda", generator=gen).bfloat16() for h in (Hq, Hkv, Hkv))
    keep = (torch.rand(R, R, device="cuda", generator=gen) < share).tril()
    mask, out = _bits(keep), torch.empty_like(q)

    def shortest(times):
        took = []
        for _ in range(times):
            begin, end = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            begin.record()
            ops.listed_attend(q, k, v, 0, mask, 128 ** -0.5, out)
            end.record()
            end.synchronize()
            took.append(begin.elapsed_time(end))
        return min(took)

    clean = shortest(6)
    v[5, :, 3] = float("inf")
    assert shortest(3) <= most * clean
    odd = ~out.isfinite()
    assert torch.equal(odd[..., 3], keep[:, 5, None].expand(R, Hq)) and not odd[..., :3].any() and not odd[..., 4:].any()


@pytest.mark.parametrize("cap,top_p,top_k,sink,window,sizes", [
    (16, 40, 200, 4, 100, (0, 16)), (16, 64, 10000, 0, 1, (8, 16)), (1, 33, 20, 2, 64, (1, 1)), (24, 17, 100, 70, 200, (0, 24)),
    (30, 10, 77, 4, 128, (3, 30)), (64, 16, 300, 4, 256, (20, 64)), (128, 8, 500, 4, 300, (0, 128)), (600, 3, 1000, 4, 64, (1, 600))])
def test_lists_as_bits_are_the_lists(cap, top_p, top_k, sink, window, sizes):
    """The bits of every row against the ids `expand` writes for it: cuts at top-k inside a bucket, empty buckets, rows before
    the first block, picks outside the table, row budgets, ids past the cache."""
    from lsa_b200 import ops

    rng = np.random.default_rng(cap)
    T, m = 1500, 60
    deal, members = rng.permutation(T), np.full((m, cap), -1, dtype=np.int32)
    at = 0
    for b in range(m):
        count = min(int(rng.integers(sizes[0], sizes[1] + 1)), T - at)
        members[b, :count] = np.sort(deal[at:at + count])
        at += count
    positions = np.concatenate([[-1, 0, 1, 5], rng.integers(0, T, 60), [T - 1]])
    R = len(positions)
    picked = np.stack([rng.permutation(m)[:top_p] if top_p <= m else rng.permutation(top_p) for _ in range(R)]).astype(np.int32)
    picked[picked >= m] = -1
    picked[3, 0] = m + 7
    picked[4:, -1] = np.where(rng.random(R - 4) < 0.5, m + 1, picked[4:, -1])  # (most of them past the cut at top-k)
    row_p = rng.integers(-1, top_p + 1, R).astype(np.int32)
    row_k = rng.integers(-1, top_k + 1, R).astype(np.int32)
    args = (cuda(picked), cuda(positions), cuda(members), top_k, sink, window)
    for budgets in ((None, None), (cuda(row_p), cuda(row_k))):
        lists, lengths, _ = ops.expand(*args, *budgets)
        for keys in (T, 1111):
            status = torch.zeros(1, dtype=torch.int32, device="cuda")
            words = ops.list_bits(*args, keys, -(-T // 128), *budgets, status=status).cpu().numpy().view(np.uint32)
            bits = np.unpackbits(words.transpose(1, 0, 2).copy().view(np.uint8), axis=-1, bitorder="little").reshape(R, -1)
            for r in range(R):
                ids = lists[r, :lengths[r]].cpu().numpy()
                assert np.array_equal(np.flatnonzero(bits[r]), np.sort(ids[ids < keys])), (r, positions[r])
            within = np.arange(top_p) < (np.full(R, top_p) if budgets[0] is None else row_p.clip(0))[:, None]
            assert int(status) == ((picked >= m) & within).sum()  # (every one, where `expand` may stop at the cut)


@pytest.mark.parametrize("cap", [112, 208, 224, 240, 400, 464, 496])
def test_a_bucket_that_ends_before_its_lanes_lends_no_key_of_the_next(cap):
    """Caps whose sixteen-place lanes, a power of two of them, pass the bucket's end: the bits are `expand`'s lists where every
    bucket of the table is full, its last one too, and no row picks two neighbours; with and without a cut at top-k."""
    from lsa_b200 import ops

    rng = np.random.default_rng(cap)
    m, R, top_p, sink, window = 9, 40, 4, 4, 64
    T = m * cap
    members = np.sort(rng.permutation(T).astype(np.int32).reshape(m, cap), axis=1)
    picked = np.stack([rng.permutation(np.arange(r % 2, m, 2))[:top_p] for r in range(R)]).astype(np.int32)
    positions = np.concatenate([[T - 1, T // 2], rng.integers(0, T, R - 2)])
    for top_k in (top_p * cap, cap + 37):
        args = (cuda(picked), cuda(positions), cuda(members), top_k, sink, window)
        lists, lengths, _ = ops.expand(*args)
        words = ops.list_bits(*args, T, -(-T // 128)).cpu().numpy().view(np.uint32)
        bits = np.unpackbits(words.transpose(1, 0, 2).copy().view(np.uint8), axis=-1, bitorder="little").reshape(R, -1)
        for r in range(R):
            assert np.array_equal(np.flatnonzero(bits[r]), np.sort(lists[r, :lengths[r]].cpu().numpy())), r


@pytest.mark.parametrize("T,Hq,Hkv,chunk,sizes", [
    (2500, 8, 2, 512, dict(pool_size=16, bucket_size=32, bucket_cap=112, cluster_block_size=512, top_p=8, top_k=300, sink_size=4,
                           window_size=300)),   # (the lanes of a bucket's bits pass its end)
    (2500, 8, 2, 512, dict(pool_size=4, bucket_size=8, bucket_cap=16, cluster_block_size=128, top_p=64, top_k=300, sink_size=4,
                           window_size=128)),   # gathered else
    (3000, 5, 1, 1024, dict(pool_size=16, bucket_size=32, bucket_cap=64, cluster_block_size=512, top_p=16, top_k=300,
                            sink_size=4, window_size=300)),  # read by bucket else
    (2000, 4, 2, 2048, dict(pool_size=16, bucket_size=64, bucket_cap=128, cluster_block_size=512, top_p=4, top_k=200,
                            sink_size=0, window_size=100))])
def test_a_prefill_read_through_masks_is_the_one_read_by_lists(T, Hq, Hkv, chunk, sizes, monkeypatch):
    """Whole prefills with the masked read for every row, up to a row inside a chunk, and for none: the same rows within the
    rounding to bf16, and no further from the gather of whole lists than that."""
    from lsa_b200 import ops
    from lsa_b200.layer import FlatDesign, FlatLayer

    rng = np.random.default_rng(T)
    w = [cuda(rng.standard_normal((Hkv * 128, 64), dtype=np.float32) / 16, torch.bfloat16) for _ in range(2)]
    layer = FlatLayer(FlatDesign(**sizes), *w, Hq, Hkv, 128)
    q, k, v = (cuda(x, torch.bfloat16) for x in layer_inputs(T, Hq, Hkv, 128, 16, T))
    listed, read = [], ops.listed_attend
    monkeypatch.setattr(ops, "listed_attend", lambda q, *a, **kw: (listed.append(q.shape[0]), read(q, *a, **kw))[1])
    gathered = layer.prefill(q, k, v, chunk=chunk, band=False, bucket_major=False).float()
    assert not listed
    for until in (0, T // 256 * 128, 128 * 1024):
        monkeypatch.setattr(FlatLayer, "_listed_until", lambda self: until)
        got = layer.prefill(q, k, v, chunk=chunk).float()
        assert bool(listed) == bool(until)
        assert (got - gathered).abs().max() <= 2e-2 and (got - gathered).abs().mean() <= 2e-3
    assert sum(listed) > T // 2
    layer.check()
    # tensors the dense read does not take go the way they went
    listed.clear()
    odd = torch.empty(T * Hq * 128 + 2, device="cuda", dtype=torch.bfloat16)[2:].view(T, Hq, 128).copy_(q)
    if sizes["bucket_cap"] <= 16:
        got = layer.prefill(odd, k, v, chunk=chunk).float()
        # (rows that no tensor map can walk are mapped in fp32: another bucket where two scores nearly tie)
        assert not listed and ((got - gathered).abs().amax((1, 2)) <= 2e-2).float().mean() >= 0.98


@pytest.mark.parametrize("short", ["masks", "picks"])
def test_a_prefill_without_memory_for_wide_masks_keeps_to_its_chunk(short, monkeypatch):
    """Where a chunk of more rows than were asked for finds no memory, for its masks or later, the rows go `chunk` at a time, and
    are the rows that they are then."""
    from lsa_b200.layer import FlatDesign, FlatLayer

    T, Hq, Hkv, chunk = 5000, 8, 2, 1024
    rng = np.random.default_rng(T)
    w = [cuda(rng.standard_normal((Hkv * 128, 64), dtype=np.float32) / 16, torch.bfloat16) for _ in range(2)]
    layer = FlatLayer(FlatDesign(pool_size=4, bucket_size=8, bucket_cap=16, cluster_block_size=128, top_p=64, top_k=300,
                                 sink_size=4, window_size=128), *w, Hq, Hkv, 128)
    q, k, v = (cuda(x, torch.bfloat16) for x in layer_inputs(T, Hq, Hkv, 128, 16, T))
    wide = layer.prefill(q, k, v, chunk=chunk).float()
    asked = []
    name = "_list_masks" if short == "masks" else "_pick"
    given = getattr(FlatLayer, name)

    def refuse(self, rows, *args):
        asked.append(rows.shape[0])
        if rows.shape[0] > chunk:
            if short == "picks":
                raise torch.OutOfMemoryError("no memory")
            return None
        return given(self, rows, *args)

    monkeypatch.setattr(FlatLayer, name, refuse)
    got = layer.prefill(q, k, v, chunk=chunk)
    assert asked[0] > chunk and max(asked[1:]) <= chunk and len(asked) > 2
    assert (got.float() - wide).abs().max() <= 2e-2 and (got.float() - wide).abs().mean() <= 2e-3
    layer.check()


@pytest.mark.parametrize("knobs", [dict(early_budget=dict(position=1500, top_k=90, top_p=20)), dict(bucket_shape=dict(rank=2, deviations=2.0)),
                                   dict(early_budget=dict(position=700, top_k=40, top_p=64), bucket_shape=dict(rank=0, deviations=1.0))])
def test_a_masked_prefill_under_an_early_budget_and_over_shaped_buckets(knobs, monkeypatch):
    """The rows' own budgets and the shaped scan in front of the masked read, against the gather of the same lists."""
    from lsa_b200 import ops
    from lsa_b200.budget import EarlyBudget
    from lsa_b200.layer import FlatDesign, FlatLayer

    T, Hq, Hkv = 2500, 8, 2
    if "early_budget" in knobs:
        knobs = dict(knobs, early_budget=EarlyBudget(**knobs["early_budget"]))
    rng = np.random.default_rng(T)
    w = [cuda(rng.standard_normal((Hkv * 128, 64), dtype=np.float32) / 16, torch.bfloat16) for _ in range(2)]
    layer = FlatLayer(FlatDesign(pool_size=4, bucket_size=8, bucket_cap=16, cluster_block_size=128, top_p=64, top_k=300,
                                 sink_size=4, window_size=128, **knobs), *w, Hq, Hkv, 128)
    q, k, v = (cuda(x, torch.bfloat16) for x in layer_inputs(T, Hq, Hkv, 128, 16, T))
    gathered = layer.prefill(q, k, v, chunk=512, band=False, bucket_major=False).float()
    listed, read = [], ops.listed_attend
    monkeypatch.setattr(ops, "listed_attend", lambda q, *a, **kw: (listed.append(q.shape[0]), read(q, *a, **kw))[1])
    got = layer.prefill(q, k, v, chunk=512).float()
    assert sum(listed) > T // 2
    assert (got - gathered).abs().max() <= 2e-2 and (got - gathered).abs().mean() <= 2e-3
    layer.check()
