"""The kernels of a decode step's few rows at the edges of their forms: the map a CTA a row, the spread expansion, the folded scan."""

import numpy as np
import pytest
import torch

from helpers import cuda, mixture, unit_rows

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


@pytest.mark.parametrize("cap,top_p,top_k,sink,window", [(1, 1024, 300, 4, 30), (31, 64, 4096, 40, 100), (33, 64, 500, 4, 64),
                                                         (256, 16, 1 << 14, 4, 700), (1030, 40, 1 << 15, 50, 64), (1280, 128, 163840, 4, 5120)])
def test_a_few_rows_list_what_many_rows_do(cap, top_p, top_k, sink, window):
    """Rows expanded a few at a time (found by samples, spread over CTAs) against the same rows among many, id for id: windows that
    cut buckets, buckets of sinks, empty and full ones, picks outside the table, budgets; positions and pages of slots."""
    from lsa_b200 import ops

    rng = np.random.default_rng(cap)
    T, m, R = 40000, 1100 if cap < 64 else 150, 5
    members = np.full((m, cap), -1, dtype=np.int32)
    for b in range(m):
        count = (0, cap, int(rng.integers(1, cap + 1)))[b % 3] if b > 4 else min(cap, 60)
        members[b, :count] = np.sort(rng.choice(T, count, replace=False)) if b > 4 else np.arange(b, 5 * count, 5)[:count]
    positions = np.array([0, 700, 20000, T - 1, 39000])
    picked = np.stack([rng.permutation(m)[:top_p] for _ in range(R)]).astype(np.int32)
    picked[:, :3] = np.array([0, 1, m + 3])[:min(3, top_p)]
    row_p, row_k = rng.integers(0, top_p + 1, R).astype(np.int32), rng.integers(0, top_k + 1, R).astype(np.int32)
    many = lambda x: None if x is None else cuda(np.concatenate([x] * 14))  # 70 rows: the other forms
    table = rng.permutation(-(-(T + 64) // 64)).astype(np.int32)
    for budgets in ((None, None), (row_p, row_k)):
        for pages in (dict(), dict(page_table=cuda(table), page_size=64)):
            for local in (True, False):
                got = ops.expand(cuda(picked), cuda(positions), cuda(members), top_k, sink, window,
                                 *(None if b is None else cuda(b) for b in budgets), local=local, **pages)
                want = ops.expand(many(picked), many(positions), cuda(members), top_k, sink, window, *(many(b) for b in budgets),
                                  local=local, **pages)
                assert torch.equal(got[0], want[0][:R]) and torch.equal(got[1], want[1][:R])
                assert 14 * int(got[2]) == int(want[2])


@pytest.mark.parametrize("m,d,keep", [(3, 64, 1), (130, 32, 128), (1024, 64, 128), (5000, 64, 33), (9001, 128, 100)])
def test_lists_folded_in_a_cluster_are_the_scan_s(m, d, keep):
    """A row's candidates split over 2 to 8 CTAs against one CTA, key for key; rows that see few or none; and a level of a tree."""
    from lsa_b200 import ops

    gen = torch.Generator(device="cuda").manual_seed(m)
    q = torch.randn(5, d, device="cuda", generator=gen)
    c = torch.randn(m, d, device="cuda", generator=gen).mul(8).round().div(8)
    c[m // 2:] = c[:m - m // 2].clone()  # (ties)
    visible = torch.tensor([m, m // 2, 1, 0, max(0, m - 1)], device="cuda", dtype=torch.int32)
    want = ops.flat_select_decode(q, c, None, visible, keep, splits=1)
    for splits in (2, 3, 7, 8):
        got = ops.flat_select_decode(q, c, None, visible, keep, splits=splits)
        assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])
    children = torch.randint(0, 1 << 20, (m, 5), device="cuda", generator=gen)
    first, end = torch.zeros_like(visible), visible
    for kids in (None, children):
        want = ops.beam_step(q, c, None, first, end, keep, children=kids, splits=1)
        for splits in (2, 8):
            got = ops.beam_step(q, c, None, first, end, keep, children=kids, splits=splits)
            assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1]) if kids is None else torch.equal(got, want)
    distinct = torch.stack([torch.randperm(m, device="cuda", generator=gen)[:min(m, 40)] for _ in range(5)]).to(torch.int32)
    none = torch.zeros_like(visible)
    want = ops.beam_step(q, c, distinct, none, none, keep, splits=1)
    got = ops.beam_step(q, c, distinct, none, none, keep, splits=8)
    assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])


@pytest.mark.parametrize("keep", [1, 31, 64, 128])
@pytest.mark.parametrize("m", [1, 255, 256, 257, 1025, 5000])
@pytest.mark.parametrize("d", [32, 64, 20])
def test_a_row_ranked_by_counting_is_the_row_scanned_whole(m, d, keep):
    """Tiles of 256 candidates that are full, ragged and empty, in one CTA, in clusters of 2 to 8 and in several clusters that are
    merged, against the scan that holds a row's best in one buffer: key for key, ties among them, rows that see few or no
    buckets, budgets, candidates named twice or not at all."""
    from lsa_b200 import ops

    gen = torch.Generator(device="cuda").manual_seed(m + d)
    q = torch.randn(6, d, device="cuda", generator=gen)
    c = torch.randn(m, d, device="cuda", generator=gen).mul(2).round().div(2)
    c[m // 2:] = c[:m - m // 2].clone()  # (ties)
    visible = torch.tensor([m, m // 2, 1, 0, max(0, m - 1), min(m, 300)], device="cuda", dtype=torch.int32)
    want = ops.flat_select(q, c, visible, keep)
    for splits in (1, 2, 5, 8, 11, 16, 32, 100):
        got = ops.flat_select_decode(q, c, None, visible, keep, splits=splits)
        assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])
        got = ops.flat_select_decode(q.repeat(3, 1), c, None, visible.repeat(3), keep, splits=splits)  # (too many for clusters)
        assert torch.equal(got[0], want[0].repeat(3, 1)) and torch.equal(got[1], want[1].repeat(3, 1))
    named = torch.randint(-1, m, (6, 300), device="cuda", generator=gen, dtype=torch.int32)
    named[:, 150:] = named[:, :150].clone()
    none = torch.zeros_like(visible)
    scores = ops.flat_select(q, c, torch.full_like(visible, m), m)[0] if m <= 512 else None
    for splits in (1, 8, 16):
        kept, keys = ops.beam_step(q, c, named, none, none, keep, splits=splits)
        for row in range(6 if scores is not None else 0):
            by_id = {0x7FFFFFFF - (int(k) & 0xFFFFFFFF): int(k) for k in scores[row].tolist()}
            best = sorted((by_id[i] for i in named[row].tolist() if i >= 0), reverse=True)[:keep]
            assert keys[row].tolist()[:len(best)] == best and set(kept[row].tolist()[len(best):]) <= {-1}


@pytest.mark.parametrize("m,d,keep,splits", [(1, 64, 3, 1), (5, 64, 128, 8), (300, 32, 64, 1), (5000, 64, 100, 32), (700, 20, 7, 8)])
def test_rows_at_their_positions_see_what_the_visible_counts_say(m, d, keep, splits):
    """The scan that counts a row's closed blocks itself, against the counts written first: positions before the first block closes,
    at a block's ends, past the table and negative."""
    from lsa_b200 import ops

    gen = torch.Generator(device="cuda").manual_seed(m)
    q, c = torch.randn(7, d, device="cuda", generator=gen), torch.randn(m, d, device="cuda", generator=gen)
    positions = torch.tensor([0, 63, 64, 127, 1 << 40, -1, -70], device="cuda")
    for block, per in ((64, 4), (64, 1), (7, 40)):
        visible = ops.visible_buckets(positions, block, per, c.shape[0])
        want = ops.flat_select_decode(q, c, None, visible, keep, splits=splits)
        got = ops.flat_select_at(q, c, positions, block, per, keep, splits=splits)
        assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])
    with pytest.raises(ValueError, match="shape"):
        ops.flat_select_at(q, c, positions, 64, 4, 129)
    with pytest.raises(ValueError, match="NULL"):  # (a table without a row)
        ops.flat_select_at(q, c[:0], positions, 64, 4, keep, splits=splits)


@pytest.mark.parametrize("rows,d_in,d_out", [(1, 2048, 64), (8, 264, 33), (3, 5120, 8), (8, 8, 1), (5, 2048, 65)])
def test_unit_rows_in_the_map_s_own_cluster(rows, d_in, d_out):
    """Maps of up to 64 columns, whose CTAs swap their columns and divide them, and a wider one in two launches: unit rows of the same
    map's plain output, in the same order of sums."""
    from lsa_b200 import ops

    gen = torch.Generator(device="cuda").manual_seed(d_in)
    x = torch.randn(rows, d_in, device="cuda", generator=gen).bfloat16()
    w = torch.randn(d_out, d_in, device="cuda", generator=gen).bfloat16()
    plain, got = ops.rows_linear(x, w), ops.rows_linear(x, w, normalize=True)
    want = plain.double() / plain.double().norm(dim=1, keepdim=True)
    assert (got.double() - want).abs().max() <= 2e-7  # (an fp32 sum of 64 squares, a root and a division)
    zero = ops.rows_linear(torch.zeros_like(x), w, normalize=True)
    assert not zero.any()


@pytest.mark.parametrize("heads,kv_heads,dh", [(40, 8, 128), (9, 1, 128), (8, 8, 64), (32, 2, 64)])
def test_a_few_rows_attend_as_many_rows_do(heads, kv_heads, dh):
    """A CTA of warps an item and its splits in a cluster, against the same rows among many (a warp an item): lists that are empty,
    shorter than a warp's stage, ragged and longer than one cluster is given, slots outside the cache, a partial read to start from.
    The probabilities are rounded to bf16 against other maxima: 2^-9 of an output's terms, which average out to a tenth of it."""
    from lsa_b200 import ops

    gen = torch.Generator(device="cuda").manual_seed(heads)
    slots, R = 9000, 7
    q = torch.randn(R, heads, dh, device="cuda", generator=gen).bfloat16()
    k, v = (torch.randn(slots, kv_heads, dh, device="cuda", generator=gen).bfloat16() for _ in range(2))
    for width in (40, 3001, 8500):
        ids = torch.stack([torch.randperm(slots + 50, device="cuda", generator=gen)[:width] for _ in range(R)]).to(torch.int32)
        lengths = torch.tensor([width, 0, 1, 31, 33, width - 1, width // 2], device="cuda", dtype=torch.int32)
        init = (torch.randn(R, heads, dh, device="cuda", generator=gen), torch.randn(R, heads, device="cuda", generator=gen))
        init[1][0, 0] = -float("inf")
        many = lambda x: torch.cat([x] * 2)
        for start in (None, init):
            want, want_lse = ops.sparse_attend(many(q), k, v, many(ids), many(lengths), dh ** -0.5, out_dtype=torch.float32,
                                               init=None if start is None else tuple(many(x) for x in start))
            for splits in (1, 2, 3, 8, 9, 16):
                got, lse = ops.sparse_attend(q, k, v, ids, lengths, dh ** -0.5, splits=splits, out_dtype=torch.float32, init=start)
                assert (got - want[:R]).abs().max() <= 2 ** -9 and (got - want[:R]).norm() <= 1e-3 * want[:R].norm()
                seen = torch.isfinite(want_lse[:R])
                assert torch.equal(torch.isfinite(lse), seen) and (lse - want_lse[:R])[seen].abs().max() <= 2e-5
                if start is None:
                    assert not got[1].any() and not seen[1].any()
            half, _ = ops.sparse_attend(q, k, v, ids, lengths, dh ** -0.5, splits=8, init=start)
            assert (half.float() - want[:R]).norm() <= 4e-3 * want[:R].norm()


@pytest.mark.parametrize("heads,kv_heads,dh", [(40, 8, 128), (9, 1, 128), (8, 8, 64), (32, 2, 64)])
@pytest.mark.parametrize("where,what", [("k", float("nan")), ("k", float("inf")), ("k", -float("inf")), ("v", float("inf")),
                                        ("v", float("nan"))])
def test_what_is_not_finite_reaches_the_few_rows_it_reaches_among_many(heads, kv_heads, dh, where, what):
    """One infinity or NaN in a listed key or value, at a list's start, in its second stage and at its end (another warp's and another
    CTA's share): the weights of zero that meet in the cluster leave what a warp an item leaves, element by element. A key of
    -inf scores -inf under half of the heads, which do not see it."""
    from lsa_b200 import ops

    gen = torch.Generator(device="cuda").manual_seed(heads)
    slots, R = 9000, 7
    q = torch.randn(R, heads, dh, device="cuda", generator=gen).bfloat16()
    k, v = (torch.randn(slots, kv_heads, dh, device="cuda", generator=gen).bfloat16() for _ in range(2))
    held = {"k": k, "v": v}[where]
    for width in (40, 3001, 8500):
        ids = torch.stack([torch.randperm(slots, device="cuda", generator=gen)[:width] for _ in range(R)]).to(torch.int32)
        lengths = torch.tensor([width, 0, 1, 31, 33, width - 1, width // 2], device="cuda", dtype=torch.int32)
        many = lambda x: torch.cat([x] * 2)
        for at in (0, 32, width - 1):
            kept = held.clone()
            held[ids[:, at].long(), 0, 3] = what
            want, want_lse = (x[:R] for x in ops.sparse_attend(many(q), k, v, many(ids), many(lengths), dh ** -0.5,
                                                               out_dtype=torch.float32))
            assert (where == "k" and abs(what) == float("inf")) or not want[0].isfinite().all()
            for splits in (2, 8, 16):
                got, lse = ops.sparse_attend(q, k, v, ids, lengths, dh ** -0.5, splits=splits, out_dtype=torch.float32)
                assert torch.equal(got.isnan(), want.isnan()) and torch.equal(got.isinf(), want.isinf()), (width, at, splits)
                finite = want.isfinite()
                assert (got - want)[finite].abs().max() <= 2 ** -9 and torch.equal(lse.isfinite(), want_lse.isfinite())
            held.copy_(kept)


@pytest.mark.parametrize("T,R,splits,sizes", [
    (700, 1, 8, dict(pool_size=4, bucket_size=8, bucket_cap=16, cluster_block_size=128, top_p=40, top_k=200, sink_size=4, window_size=128)),
    (9000, 8, 1, dict(pool_size=16, bucket_size=32, bucket_cap=64, cluster_block_size=256, top_p=64, top_k=700, sink_size=0, window_size=100)),
    # (lists out of the scan itself up to eight ids a thread, and one id past that: 127 picks of 128 and the window)
    (20000, 3, 8, dict(pool_size=4, bucket_size=64, bucket_cap=128, cluster_block_size=512, top_p=127, top_k=3000, sink_size=40,
                       window_size=128)),
    (20000, 8, 8, dict(pool_size=4, bucket_size=64, bucket_cap=128, cluster_block_size=512, top_p=127, top_k=9000, sink_size=3,
                       window_size=129))])
def test_a_step_in_one_call_is_the_calls_it_is_made_of(T, R, splits, sizes, monkeypatch):
    """The same rows bit for bit, at the end, in the middle and before the first block; strided queries; a status that is raised. Lists
    that the scan writes itself are the expansion's."""
    from helpers import layer_inputs
    from lsa_b200 import ops
    from lsa_b200.layer import FlatDesign, FlatLayer

    rng = np.random.default_rng(T)
    w = [cuda(rng.standard_normal((256, 64), dtype=np.float32) / 16, torch.bfloat16) for _ in range(2)]
    layer = FlatLayer(FlatDesign(**sizes), *w, 8, 2, 128)
    q, k, v = (cuda(x, torch.bfloat16) for x in layer_inputs(T, 8, 2, 128, 16, T))
    index = layer.build_index(k)
    positions = cuda(np.array([T - 1, T // 2, 5, 0, 130, T - 2, 256, 90])[:R])
    once, calls = ops.flat_decode, []
    monkeypatch.setattr(ops, "flat_decode", lambda *a: (calls.append(1), once(*a))[1])
    for rows in (q[positions], q.repeat(1, 2, 1)[positions][:, :8]):
        got = layer.decode(rows, positions, k, v, index, splits=splits)
        with monkeypatch.context() as patch:
            patch.setattr(FlatLayer, "_decodes_in_one_call", lambda *a: False)
            assert torch.equal(got, layer.decode(rows, positions, k, v, index, splits=splits))
    assert len(calls) == 2
    layer.decode(q[positions], positions.int(), k, v, index)  # (positions that would be converted: the calls one by one)
    assert len(calls) == 2
    layer.check()


@pytest.mark.parametrize("m,cap,top_p,top_k,window,sink", [(1024, 64, 64, 3000, 128, 4), (1024, 1, 1, 1, 1, 0),
                                                            (1000, 1280, 128, 163840, 5120, 4), (4100, 33, 127, 1000, 50, 40),
                                                            (300, 128, 127, 9000, 128, 0), (300, 128, 127, 9000, 129, 0), (40, 7, 9, 60, 3, 2)])
def test_lists_out_of_the_scan_are_the_expansion_s_of_its_picks(m, cap, top_p, top_k, window, sink):
    """One to nine rows over one CTA, a cluster and several, before the first block, at its end and at the last; lists out of the scan
    itself (2,048 ids a CTA at most), of an expansion that merges, and of the calls one after another: the same ids."""
    from lsa_b200 import ops

    gen = torch.Generator(device="cuda").manual_seed(m + cap)
    per, block = 10, 10 * cap
    q, c = (torch.nn.functional.normalize(torch.randn(n, 64, device="cuda", generator=gen), dim=-1) for n in (9, m))
    c[m // 2:m // 2 + 5] = c[:5]  # (ties)
    bucket, place = torch.arange(m, device="cuda")[:, None], torch.arange(cap, device="cuda")
    members = (bucket // per * block + bucket % per + place * per).to(torch.int32)
    members[torch.rand(m, cap, device="cuda", generator=gen).sort(-1, descending=True).values < 0.2] = -1  # (ragged: pads at the end)
    last = m * cap - 1
    positions = torch.tensor([last, 0, block - 1, block, last // 2, last // 3, 3 * block + 5, last - 1, block * (m // per)], device="cuda")
    for rows in (1, 3, 8, 9):
        for splits in (1, 2, 8, 15, 16, 32):
            _, picked = ops.flat_select_at(q[:rows], c, positions[:rows], block, per, top_p, splits=splits)
            want, lengths, _ = ops.expand(picked, positions[:rows], members, top_k, sink, window)
            got, got_lengths = ops.flat_lists_at(q[:rows], c, positions[:rows], block, per, members, top_p, top_k, sink, window,
                                                 splits=splits)
            assert torch.equal(got_lengths, lengths)
            seen = torch.arange(want.shape[1], device="cuda") < lengths[:, None]
            assert torch.equal(torch.where(seen, got, -1), torch.where(seen, want, -1))
    with pytest.raises(ValueError):  # (128 picks at most)
        ops.flat_lists_at(q, c, positions, block, per, members, 129, top_k, sink, window)


def test_a_step_before_the_first_block_has_closed_is_refused_either_way(monkeypatch):
    """An index without a bucket (a cache shorter than a cluster block): the scan of a few rows takes no empty table, in one call
    or one by one."""
    from helpers import layer_inputs
    from lsa_b200.layer import FlatDesign, FlatLayer

    w = [cuda(np.zeros((256, 64), dtype=np.float32), torch.bfloat16) for _ in range(2)]
    layer = FlatLayer(FlatDesign(pool_size=4, bucket_size=8, bucket_cap=16, cluster_block_size=128, top_p=40, top_k=200,
                                 sink_size=4, window_size=32), *w, 8, 2, 128)
    q, k, v = (cuda(x, torch.bfloat16) for x in layer_inputs(100, 8, 2, 128, 16, 100))
    index, positions = layer.build_index(k), cuda(np.array([99, 50]))
    for once in (True, False):
        monkeypatch.setattr(FlatLayer, "_decodes_in_one_call", lambda *a: once)
        with pytest.raises(ValueError, match="NULL"):
            layer.decode(q[positions], positions, k, v, index)


@pytest.mark.parametrize("rows", [129, 700, 19000])  # (32 rows a CTA, and 64)
@pytest.mark.parametrize("d_in,d_idx", [(256, 32), (192, 64), (130, 64), (64, 60), (256, 128), (100, 100)])
def test_the_exact_map_keeps_the_oracle_s_bits(rows, d_in, d_idx):
    """Whole slices of input and output dims and ragged ones, against the oracle's product in its own order, bit for bit."""
    from lsa_b200 import ops

    rng = np.random.default_rng(d_in + d_idx)
    x, w = rng.standard_normal((rows, d_in), dtype=np.float32), rng.standard_normal((d_in, d_idx), dtype=np.float32)
    got = ops.index_map(cuda(x)[:, None], cuda(w), normalize=False).cpu().numpy()
    some = np.unique(np.concatenate([np.arange(40), rng.integers(0, rows, 60), np.arange(rows - 40, rows)]))
    want = np.zeros((len(some), d_idx), dtype=np.float32)
    for k in range(d_in):  # (a multiply-add in 64 bits rounds to the fp32 one: 48 bits of product beside 24)
        want = (x[some, k, None].astype(np.float64) * w[k].astype(np.float64) + want.astype(np.float64)).astype(np.float32)
    off = got[some].view(np.int32).astype(np.int64) - want.view(np.int32)
    assert (off == 0).mean() >= 0.999 and np.abs(got[some] - want).max() <= 1e-4  # (a double rounding in a million)


@pytest.mark.parametrize("G,P,d", [(1, 1025, 64), (16, 640, 32), (20, 520, 64), (32, 640, 16), (5, 4096, 16)])
def test_ward_over_clusters_and_over_a_grid_keeps_the_oracle_s_labels(oracle, G, P, d):
    """Blocks past one CTA's shared memory as grids of 148, 9, 7 and 29 CTAs a block and as clusters of four, in turn on the same
    workspace (the counters of arrivals are set up by every call), and replayed from a graph."""
    from lsa_b200 import ops

    keys = unit_rows(mixture(G * P, d, 24, 0.4, G + P)).reshape(G, P, d)
    count = (P + 1) // 2  # (pairs, and the one left over)
    want, want_reached, want_rounds = oracle.ward_rounds(keys, np.ones((G, P), dtype=np.float32), count, 2.0, return_rounds=True)
    pools, workspace = cuda(keys), torch.full((64 << 20,), 255, device="cuda", dtype=torch.uint8)
    for _ in range(2):
        got, reached, rounds = ops.ward_rounds(pools, 1.0, count, 2.0, return_rounds=True, workspace=workspace)
        assert np.array_equal(got.cpu().numpy(), want) and np.array_equal(rounds.cpu().numpy(), want_rounds)
        assert np.array_equal(reached.cpu().numpy(), want_reached)
    labels, flags = torch.empty_like(got), torch.empty(G, device="cuda", dtype=torch.uint8)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        ops.ward_rounds(pools, 1.0, count, 2.0, labels=labels, reached=flags, workspace=workspace)
    for _ in range(2):
        labels.fill_(-1)
        graph.replay()
        assert np.array_equal(labels.cpu().numpy(), want) and np.array_equal(flags.bool().cpu().numpy(), want_reached)
