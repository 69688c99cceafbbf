"""Parity of every CUDA kernel with the CPU oracle, called through the C ABI (via the ctypes wrappers).

Integer results (labels, member tables, picked buckets, read lists) must be bit-exact. Floats: index vectors within
2e-6 (fp32 sums in another order), attention within max-abs 2e-2 / mean-abs 2e-3 of the fp32 oracle on bf16 inputs.
"""

import threading

import numpy as np
import pytest
import torch

from conftest import golden
from helpers import bf16_round, cuda, layer_inputs, mixture, unit_rows

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ops():
    from lsa_b200 import ops as module

    return module


# ------------------------------------------------------------------------------------------------ index map


@pytest.mark.parametrize("T,Hq,Hkv,dh,d_idx", [(300, 8, 2, 128, 32), (1000, 40, 8, 128, 64), (65, 4, 4, 64, 16)])
def test_index_map_matches_the_oracle(ops, oracle, T, Hq, Hkv, dh, d_idx):
    q, k, _ = layer_inputs(T, Hq, Hkv, dh, 8, 0)
    rng = np.random.default_rng(1)
    w = bf16_round(rng.standard_normal((Hkv * dh, d_idx), dtype=np.float32) / np.sqrt(Hkv * dh))
    want_q = oracle.project(oracle.regroup_queries(q, Hkv), w)
    want_k = oracle.project(k.reshape(T, -1), w)
    got_q, got_q16 = ops.index_map(cuda(q, torch.bfloat16), cuda(w, torch.bfloat16), group=Hq // Hkv, also_bf16=True)
    got_k = ops.index_map(cuda(k, torch.bfloat16), cuda(w), group=1)
    np.testing.assert_allclose(got_q.cpu().numpy(), want_q, rtol=0, atol=2e-6)
    np.testing.assert_allclose(got_k.cpu().numpy(), want_k, rtol=0, atol=2e-6)
    np.testing.assert_allclose(got_q16.float().cpu().numpy(), want_q, rtol=0, atol=4e-3)


@pytest.mark.parametrize("T,Hq,Hkv,dh,d_idx,off", [(1000, 40, 8, 128, 64, 0), (333, 8, 2, 128, 32, 0),
                                                     (4100, 16, 4, 64, 128, 16)])
def test_tensor_core_map_matches_the_oracle(ops, oracle, T, Hq, Hkv, dh, d_idx, off):
    q, k, _ = layer_inputs(T, Hq, Hkv, dh, 8, 5)
    rng = np.random.default_rng(2)
    used = dh - off
    w = bf16_round(rng.standard_normal((Hkv * used, d_idx), dtype=np.float32) / np.sqrt(Hkv * used))
    want_q = oracle.project(oracle.regroup_queries(q[:, :, off:], Hkv), w)
    want_k = oracle.project(np.ascontiguousarray(k[:, :, off:]).reshape(T, -1), w)
    W = cuda(w, torch.bfloat16)
    wq_t = ops.expand_map(W, Hq, Hq // Hkv, dh, off)
    wk_t = ops.expand_map(W, Hkv, 1, dh, off)
    assert wq_t.shape == (d_idx, Hq * dh) and wk_t.shape == (d_idx, Hkv * dh)
    status = torch.zeros(1, dtype=torch.int32).cuda()
    got_q = ops.index_map_tc(cuda(q, torch.bfloat16), wq_t, status=status)
    got_k = ops.index_map_tc(cuda(k, torch.bfloat16), wk_t, status=status)
    assert int(status) == 0
    np.testing.assert_allclose(got_q.cpu().numpy(), want_q, rtol=0, atol=3e-5)
    np.testing.assert_allclose(got_k.cpu().numpy(), want_k, rtol=0, atol=3e-5)
    # it agrees with the exact-order kernel to the same bound, and not normalising leaves the raw product
    exact = ops.index_map(cuda(q, torch.bfloat16), W, group=Hq // Hkv, dh_off=off)
    assert (exact - got_q).abs().max() <= 3e-5
    raw = ops.index_map_tc(cuda(k, torch.bfloat16), wk_t, normalize=False)
    want_raw = oracle.project(np.ascontiguousarray(k[:, :, off:]).reshape(T, -1), w, normalize=False)
    np.testing.assert_allclose(raw.cpu().numpy(), want_raw, rtol=1e-4, atol=1e-4)


def test_two_layer_map_matches_its_restatement(ops, oracle):
    """A variant with no reference code: the oracle restatement is the only pin."""
    from scipy.special import erf

    rng = np.random.default_rng(3)
    T, d_in, d_hidden, d_idx = 700, 128, 2048, 64
    x = bf16_round(rng.standard_normal((T, d_in), dtype=np.float32))
    w1 = bf16_round(rng.standard_normal((d_in, d_hidden), dtype=np.float32) / np.sqrt(d_in))
    w2 = bf16_round(rng.standard_normal((d_hidden, d_idx), dtype=np.float32) / np.sqrt(d_hidden))
    got = ops.mlp_map(cuda(x, torch.bfloat16), cuda(w1.T.copy(), torch.bfloat16), cuda(w2.T.copy(), torch.bfloat16))
    # the kernel keeps the hidden layer in bf16: restate with that rounding, then against the pure fp32 form
    pre = oracle.project(x, w1, normalize=False)
    hidden = bf16_round(0.5 * pre * (1.0 + erf(pre * np.float32(0.7071067811865476))))
    np.testing.assert_allclose(got.cpu().numpy(), oracle.project(hidden, w2), rtol=0, atol=2e-4)
    np.testing.assert_allclose(got.cpu().numpy(), oracle.project_mlp(x, w1, w2), rtol=0, atol=3e-3)


def test_index_map_identity_zero_rows_and_rotary_offsets(ops, oracle):
    g = golden("index_space")
    q, k = cuda(g["q"]), cuda(g["k"])
    iq = ops.index_map(q, None, group=4)
    ik = ops.index_map(k, None, group=1)
    np.testing.assert_allclose(iq.cpu().numpy(), g["index_queries"], rtol=0, atol=2e-6)
    np.testing.assert_allclose(ik.cpu().numpy(), g["index_keys"], rtol=0, atol=2e-6)
    assert not ik[7].any()
    proj = ops.index_map(ik[:, None, :], cuda(g["w"]))
    np.testing.assert_allclose(proj.cpu().numpy(), g["projected_keys"], rtol=0, atol=2e-6)
    # the rotary prefix dropped: dims 8.. of every head
    part = ops.index_map(k, None, group=1, dh_off=8, normalize=False)
    assert torch.equal(part, k[:, :, 8:].reshape(k.shape[0], -1))


# ------------------------------------------------------------------------------------------------ pooling, Ward, table


def test_pooling_is_bit_exact(ops, oracle):
    keys = unit_rows(mixture(4096, 64, 16, 0.3, 3))
    want = oracle.pool_keys(keys.reshape(8, 512, 64), 16)
    got = ops.pool_keys(cuda(keys).view(8, 512, 64), 16)
    assert np.array_equal(got.cpu().numpy().view(np.int32), want.view(np.int32))
    got16 = ops.pool_keys(cuda(keys, torch.bfloat16).view(8, 512, 64), 16)
    want16 = oracle.pool_keys(bf16_round(keys).reshape(8, 512, 64), 16)
    assert np.array_equal(got16.cpu().numpy().view(np.int32), want16.view(np.int32))


@pytest.mark.parametrize("G,P,d,pool,count,cap", [(6, 64, 64, 16, 32, 64), (3, 256, 64, 4, 64, 32),
                                                   (4, 80, 64, 64, 8, 1280), (5, 32, 16, 4, 16, 16),
                                                   (2, 64, 48, 4, 16, 24), (2, 512, 64, 2, 64, 32)])
def test_ward_labels_are_bit_exact(ops, oracle, G, P, d, pool, count, cap):
    keys = unit_rows(mixture(G * P * pool, d, 12, 0.3, P + d))
    pools = oracle.pool_keys(keys.reshape(G, P * pool, d), pool)
    sizes = np.full((G, P), float(pool), dtype=np.float32)
    want, want_reached, want_rounds = oracle.ward_rounds(pools, sizes, count, cap, return_rounds=True)
    got, reached, rounds = ops.ward_rounds(cuda(pools), float(pool), count, cap, return_rounds=True)
    assert np.array_equal(got.cpu().numpy(), want)
    assert np.array_equal(reached.cpu().numpy(), want_reached)
    assert np.array_equal(rounds.cpu().numpy(), want_rounds)
    got2, _ = ops.ward_rounds(cuda(pools), cuda(sizes), count, cap)
    assert torch.equal(got, got2)


@pytest.mark.parametrize("G,P,d,count,cap,sizes", [(3, 1024, 64, 512, 2.0, 1.0), (2, 2048, 16, 1024, 2.0, 1.0),
                                                     (2, 768, 64, 96, 64.0, 4.0), (1, 640, 32, 600, 2.0, 1.0)])
def test_large_block_ward_is_bit_exact(ops, oracle, G, P, d, count, cap, sizes):
    """Blocks past one CTA's shared memory: the multi-launch merge (the tree's pairings at a cap of two, and a
    general cap), against the oracle label for label and round for round."""
    keys = unit_rows(mixture(G * P, d, 40, 0.4, P + d)).reshape(G, P, d) * np.float32(3.0)
    size_rows = np.full((G, P), sizes, dtype=np.float32)
    want, want_reached, want_rounds = oracle.ward_rounds(keys, size_rows, count, cap, return_rounds=True)
    got, reached, rounds = ops.ward_rounds(cuda(keys), sizes, count, cap, return_rounds=True)
    assert np.array_equal(got.cpu().numpy(), want)
    assert np.array_equal(reached.cpu().numpy(), want_reached)
    assert np.array_equal(rounds.cpu().numpy(), want_rounds)


@pytest.mark.parametrize("G,P,d,count,cap,sizes", [(7, 1, 64, 1, 8.0, 1.0), (3, 5, 32, 2, 8.0, 1.0), (1, 65, 64, 8, 640.0, 64.0),
                                                     (9, 128, 64, 64, 16.0, 4.0), (150, 96, 16, 12, 64.0, 4.0),
                                                     (2, 512, 64, 64, 32.0, 2.0), (2, 513, 64, 257, 2.0, 1.0),
                                                     (80, 640, 16, 320, 2.0, 1.0), (1, 4096, 64, 2048, 2.0, 1.0)])
def test_ward_blocks_over_one_to_eight_ctas_are_bit_exact(ops, oracle, G, P, d, count, cap, sizes):
    """One pool, a ragged second tile, blocks of a CTA and of a cluster, key sums in shared memory up to 512 pools and in
    the workspace above, both tile heights; and sizes that differ, so that rows close at different times."""
    keys = unit_rows(mixture(G * P, d, 24, 0.4, G + P + d)).reshape(G, P, d) * np.float32(2.0)
    rng = np.random.default_rng(P)
    for size_rows in (np.full((G, P), sizes, dtype=np.float32), sizes * rng.integers(1, 4, (G, P)).astype(np.float32)):
        want, want_reached, want_rounds = oracle.ward_rounds(keys, size_rows, count, cap, return_rounds=True)
        got, reached, rounds = ops.ward_rounds(cuda(keys), cuda(size_rows), count, cap, return_rounds=True)
        assert np.array_equal(got.cpu().numpy(), want)
        assert np.array_equal(reached.cpu().numpy(), want_reached)
        assert np.array_equal(rounds.cpu().numpy(), want_rounds)


@pytest.mark.parametrize("G,whole,tile", [(150, 64, 64), (80, 512, 128)])
@pytest.mark.parametrize("quarters", [(0, 1), (1, 0), (1, 1), (2, 0), (2, 1), (4, -1)])
def test_ward_of_a_last_row_tile_with_few_rows_is_bit_exact(ops, oracle, G, whole, tile, quarters):
    """A last row tile of one row, of up to two rows a warp, of up to four and of more, beside whole ones, the partners' tiles ragged
    the same way; later rounds leave tiles that are part dirty and part steady."""
    P = whole + quarters[0] * tile // 4 + quarters[1]
    keys = unit_rows(mixture(G * P, 16, 24, 0.4, P)).reshape(G, P, 16) * np.float32(2.0)
    size_rows = np.full((G, P), 4.0, dtype=np.float32)
    want, want_reached, want_rounds = oracle.ward_rounds(keys, size_rows, P // 4, 32.0, return_rounds=True)
    got, reached, rounds = ops.ward_rounds(cuda(keys), 4.0, P // 4, 32.0, return_rounds=True)
    assert np.array_equal(got.cpu().numpy(), want)
    assert np.array_equal(reached.cpu().numpy(), want_reached) and np.array_equal(rounds.cpu().numpy(), want_rounds)


@pytest.mark.parametrize("scale", [1e-30, 1e-22, 1e-19, 3e-17, 1e-10, 1e14, 1e15, 4e18, 1.2e19])
@pytest.mark.parametrize("P", [96, 600])
def test_ward_of_keys_whose_squares_leave_fp32s_range_is_bit_exact(ops, oracle, scale, P):
    """Norms whose squares are denormal, zero or infinite, in both forms: the costs are the replay's, so the labels are."""
    rng = np.random.default_rng(P)
    with np.errstate(all="ignore"):
        keys = (unit_rows(mixture(2 * P, 64, 12, 0.4, P)) * rng.uniform(0.3, 2.0, (2 * P, 1)) * scale).astype(np.float32)
        keys = keys.reshape(2, P, 64)
        sizes = np.full((2, P), 4.0, np.float32)
        want, want_reached, want_rounds = oracle.ward_rounds(keys, sizes, P // 8, 64.0, return_rounds=True)
    got, reached, rounds = ops.ward_rounds(cuda(keys), cuda(sizes), P // 8, 64.0, return_rounds=True)
    assert np.array_equal(got.cpu().numpy(), want)
    assert np.array_equal(reached.cpu().numpy(), want_reached) and np.array_equal(rounds.cpu().numpy(), want_rounds)


def test_ward_golden_and_adversarial_cases(ops, oracle):
    g = golden("ward")
    for tag in "abcde":
        pool, count, cap = g[f"{tag}_args"].tolist()
        labels, reached = ops.ward_rounds(cuda(g[f"{tag}_pools"]), float(pool), count, cap)
        assert reached.all() and np.array_equal(labels.cpu().numpy(), g[f"{tag}_labels"])
    four = torch.full((1, 4), 4.0).cuda()
    assert ops.ward_rounds(cuda(g["tight_pools"]), four, 3, 16)[0].tolist() == [[0, 0, 1, 2]]
    assert ops.ward_rounds(cuda(g["same_pools"]), four, 2, 16)[0].tolist() == [[0, 0, 0, 1]]
    labels, reached = ops.ward_rounds(cuda(g["pair_pools"]), 1.0, 32, 2)
    assert reached.all() and np.array_equal(labels.cpu().numpy(), g["pair_labels"])
    # near-copied and rounded pools (ties everywhere): bit-exact with the oracle, which runs the same order
    for tag in ("near", "rounded"):
        pools = g[f"{tag}_pools"]
        want, want_reached = oracle.ward_rounds(pools, np.full(pools.shape[:2], 4.0, np.float32), 64, 16)
        got, reached = ops.ward_rounds(cuda(pools), 4.0, 64, 16)
        assert np.array_equal(got.cpu().numpy(), want) and np.array_equal(reached.cpu().numpy(), want_reached)
    # a cap that leaves no pair: every pool stays alone and the block reports short
    sixteen = cuda(g["b_pools"][:2, :16])
    labels, reached = ops.ward_rounds(sixteen, 16.0, 8, 16)
    assert not reached.any() and torch.equal(labels.cpu(), torch.arange(16).expand(2, 16))


@pytest.mark.parametrize("cap,m,top_p,top_k,rows", [(1, 90, 70, 33, 70), (16, 300, 130, 900, 70), (17, 200, 64, 500, 9),
                                                     (63, 80, 33, 2079, 70), (64, 80, 40, 700, 70), (65, 128, 128, 8320, 70),
                                                     (100, 90, 90, 2000, 70), (1280, 40, 30, 20000, 65)])
def test_lists_over_narrow_and_wide_buckets_are_the_oracles(ops, oracle, cap, m, top_p, top_k, rows):
    """Picks walked as one run of places (up to 64 members a bucket), a CTA a row over runs of members (wider buckets, long
    lists) and a warp a row: ragged and empty buckets, empty picks, the cut inside a pick, window and sinks, rows at early
    positions, a row's own budgets, and an owner's range."""
    rng = np.random.default_rng(cap * 7 + m)
    sizes = rng.integers(0, cap + 1, m)
    order = rng.permutation(m * cap).astype(np.int32)
    members, at = np.full((m, cap), -1, np.int32), 0
    for b in range(m):
        members[b, :sizes[b]] = np.sort(order[at:at + sizes[b]])
        at += sizes[b]
    picked = np.stack([rng.permutation(m)[:top_p] if top_p <= m else np.r_[rng.permutation(m), -np.ones(top_p - m)]
                       for _ in range(rows)]).astype(np.int32)
    picked[rng.random(picked.shape) < 0.1] = -1
    positions = rng.integers(0, m * cap + 50, rows)
    positions[:3] = 0, 1, m * cap + 40
    for sink, window in ((0, 1), (4, 37)):
        want, want_len = oracle.expand(picked, positions, members, top_k, sink, window)
        got, lens, status = ops.expand(cuda(picked), cuda(positions), cuda(members), top_k, sink, window)
        assert np.array_equal(got.cpu().numpy(), want) and np.array_equal(lens.cpu().numpy(), want_len) and not int(status)
    cut = int(np.median(positions))
    want, want_len = oracle.expand(picked, positions, members, top_k, 4, 37, early_budget=(cut, top_k // 3 + 1, top_p // 2 + 1))
    early = cuda(positions) < cut
    row_p = torch.where(early, top_p // 2 + 1, top_p).to(torch.int32)
    row_k = torch.where(early, top_k // 3 + 1, top_k).to(torch.int32)
    got, lens, _ = ops.expand(cuda(picked), cuda(positions), cuda(members), top_k, 4, 37, row_p, row_k)
    assert np.array_equal(got.cpu().numpy(), want) and np.array_equal(lens.cpu().numpy(), want_len)
    half = m * cap // 2
    parts = [ops.expand(cuda(picked), cuda(positions), cuda(members), top_k, 4, 37, row_p, row_k, owner=owner)[:2]
             for owner in ((0, half), (half, 1 << 40))]
    for r in range(rows):
        ids = want[r][:want_len[r]]
        for (lists, lengths), mine in zip(parts, (ids < half, ids >= half)):
            assert np.array_equal(lists[r].cpu().numpy()[:int(lengths[r])], ids[mine])


@pytest.mark.parametrize("rows,cap,top_p", [(70, 16, 40), (70, 65, 20), (70, 100, 90), (5, 64, 40), (5, 1280, 40)])
def test_rows_before_the_first_position_and_empty_budgets_have_empty_lists(ops, rows, cap, top_p):
    """Every form of the expansion (a warp, a CTA or a cluster a row): nothing is listed, and nothing written outside the row."""
    m, top_k, sink, window = 100, 500, 4, 32
    members = cuda(np.arange(m * cap, dtype=np.int32).reshape(m, cap))
    picked = cuda(np.stack([np.random.default_rng(r).permutation(m)[:top_p] for r in range(rows)]).astype(np.int32))
    width = top_k + window + sink
    for position, p_row, k_row in ((-1, 9, 9), (-5, 9, 9), (-1000, 9, 9), (3000, 9, -5), (3000, -3, 9), (3000, 0, 0)):
        positions = torch.full((rows,), position, device="cuda", dtype=torch.int64)
        budgets = [torch.full((rows,), x, device="cuda", dtype=torch.int32) for x in (p_row, k_row)]
        room = torch.full((rows + 8, width), 123, device="cuda", dtype=torch.int32)
        lengths, status = (torch.zeros(n, device="cuda", dtype=torch.int32) for n in (rows, 1))
        ops.expand(picked, positions, members, top_k, sink, window, *budgets, outs=(room[4:-4], lengths, status))
        local = min(max(position + 1, 0), window + sink)
        assert (lengths == local).all() and (room[:4] == 123).all() and (room[-4:] == 123).all()
        want = [*range(position + 1 - window, position + 1), *range(sink)][:local]
        assert all(row == want + [-1] * (width - local) for row in room[4:-4].tolist())


def test_linear_layers_over_a_few_rows(ops):
    """The decode-row maps: heads summed or read side by side, GELU or not, unit rows or not, against fp32 torch on
    the same bf16 values (the hidden layer of the two-layer map is rounded to bf16, as the batched map rounds it)."""
    gen = torch.Generator().manual_seed(3)
    for rows in (1, 3, 8):
        x = (0.5 * torch.randn(rows, 64, 576, generator=gen)).bfloat16().cuda()
        w1 = (torch.randn(2048, 576, generator=gen) / 24).bfloat16().cuda()
        w2 = (torch.randn(64, 2048, generator=gen) / 45).bfloat16().cuda()
        summed = x.float().sum(1).bfloat16().float()
        want_hidden = torch.nn.functional.gelu(summed @ w1.float().t())
        hidden = ops.rows_linear(x, w1, sum_heads=True, gelu=True, out_dtype=torch.bfloat16)
        assert (hidden.float() - want_hidden).abs().max() <= 2e-2 * want_hidden.abs().max()
        want = torch.nn.functional.normalize(hidden.float() @ w2.float().t(), dim=1)
        got = ops.rows_linear(hidden, w2, normalize=True)
        assert (got - want).abs().max() <= 1e-5
        # heads side by side under a widened map: [rows, 40, 128] against [64, 5120]
        q = torch.randn(rows, 40, 128, generator=gen).bfloat16().cuda()
        wide = (torch.randn(64, 5120, generator=gen) / 70).bfloat16().cuda()
        got = ops.rows_linear(q, wide, normalize=True)
        want = torch.nn.functional.normalize(q.float().reshape(rows, -1) @ wide.float().t(), dim=1)
        assert (got - want).abs().max() <= 1e-5
        plain = ops.rows_linear(q, wide)
        assert (plain - q.float().reshape(rows, -1) @ wide.float().t()).abs().max() <= 1e-4
    with pytest.raises(ValueError):
        ops.rows_linear(torch.zeros(9, 64, device="cuda", dtype=torch.bfloat16), wide)


def test_a_rows_gather_does_not_depend_on_the_rows_beside_it(ops):
    """Items are spread one warp a CTA while there are fewer than SMs, up to seven a CTA: the same bits either way."""
    gen = torch.Generator(device="cuda").manual_seed(11)
    for Hq, Hkv, dh in ((8, 2, 128), (24, 2, 128), (8, 2, 64)):
        q = torch.randn(260, Hq, dh, generator=gen, device="cuda").bfloat16()
        k, v = (torch.randn(900, Hkv, dh, generator=gen, device="cuda").bfloat16() for _ in range(2))
        ids = torch.stack([torch.randperm(900, generator=gen, device="cuda")[:333] for _ in range(260)]).to(torch.int32)
        lens = torch.randint(0, 334, (260,), generator=gen, device="cuda", dtype=torch.int32)
        for splits in (1, 3, 16):
            whole, whole_lse = ops.sparse_attend(q, k, v, ids, lens, dh ** -0.5, splits=splits)
            for n in (1, 5, 80):
                part, lse = ops.sparse_attend(q[:n], k, v, ids[:n], lens[:n], dh ** -0.5, splits=splits)
                if splits == 1:
                    assert torch.equal(part, whole[:n]) and torch.equal(lse, whole_lse[:n])
                else:  # (the merge of the splits goes by the number of rows: fp32 sums of up to 16 terms, rounded to bf16)
                    assert (part.float() - whole[:n].float()).abs().max() <= 2 ** -8 * whole.float().abs().max()


def test_kmeans_bucketing_matches_its_restatement(ops, oracle):
    """A variant with no reference code: config 1's shapes - 1,024 pools, 256 centres, 32 dims, 10 rounds."""
    keys = unit_rows(mixture(16384, 32, 64, 0.3, 8))
    pools = oracle.pool_keys(keys[None], 16)[0]
    rng = np.random.default_rng(0)
    init = unit_rows(pools[rng.permutation(len(pools))[:256]])
    want_centroids, want_assign = oracle.kmeans(pools, init, 10)
    centroids, assign = ops.kmeans(cuda(pools), cuda(init), 10)
    assert np.array_equal(assign.cpu().numpy(), want_assign)
    assert np.array_equal(centroids.cpu().numpy().view(np.int32), want_centroids.view(np.int32))


@pytest.mark.parametrize("G,P,pool,count,cap", [(1, 33, 3, 5, 40), (2, 2049, 1, 1024, 3), (700, 40, 2, 8, 8), (1, 5000, 1, 7, 900)])
def test_bucket_table_of_ragged_blocks(ops, G, P, pool, count, cap):
    """Pools past a step of the walk, buckets over their cap (cut, and counted), labels past the table (left out), one
    bucket a CTA and many: against the walk as written."""
    rng = np.random.default_rng(P)
    labels = rng.integers(0, count + 1, (G, P))
    keys = rng.standard_normal((G * P * pool, 32), dtype=np.float32)
    members, sizes, sums, cent, _, status = ops.bucket_table(cuda(keys), cuda(labels), pool, count, cap)
    want, over = np.full((G * count, cap), -1, np.int32), 0
    for g in range(G):
        for b in range(count):
            ids = (g * P * pool + np.flatnonzero(labels[g] == b)[:, None] * pool + np.arange(pool)).reshape(-1)
            over += len(ids) > cap
            want[g * count + b, :min(len(ids), cap)] = ids[:cap]
    assert np.array_equal(members.cpu().numpy(), want) and int(status) == over
    assert np.array_equal(sizes.cpu().numpy(), (want >= 0).sum(1))
    for row in rng.integers(0, G * count, 20):  # added one by one, ascending: fp32, so equal and not close
        acc = np.zeros(32, np.float32)
        for i in want[row][want[row] >= 0]:
            acc = acc + keys[i]
        assert np.array_equal(sums.cpu().numpy()[row], acc)


def test_bucket_table_of_the_widest_keys(ops):
    """One bucket whose sums and norm are all of a CTA's shared memory, as this call has always taken: 58,111 dims."""
    gen = torch.Generator(device="cuda").manual_seed(5)
    keys = torch.randn(3, 58111, generator=gen, device="cuda")
    members, sizes, sums, cent, _, status = ops.bucket_table(keys, torch.zeros(1, 3, device="cuda", dtype=torch.int64), 1, 1, 4)
    assert members.tolist() == [[0, 1, 2, -1]] and sizes.tolist() == [3] and not int(status)
    assert torch.equal(sums[0], (keys[0] + keys[1]) + keys[2])
    assert (cent[0].norm() - 1).abs() <= 1e-3  # (58,111 squares added one by one: 58,111 * 2^-24 of the sum at most)
    with pytest.raises(ValueError):
        ops.bucket_table(torch.zeros(3, 58112, device="cuda"), torch.zeros(1, 3, device="cuda", dtype=torch.int64), 1, 1, 4)


def test_bucket_table_is_bit_exact(ops, oracle):
    for name, (pool, bucket, cap, block) in {"flat_small": (4, 8, 16, 64), "flat_c1like": (16, 64, 128, 512)}.items():
        g = golden(name)
        want = oracle.build_buckets(g["keys"], pool, bucket, cap, block)
        G = g["keys"].shape[0] // block
        pools = oracle.pool_keys(g["keys"][: G * block].reshape(G, block, -1), pool)
        labels, _ = oracle.ward_rounds(pools, np.full(pools.shape[:2], float(pool), np.float32), block // bucket, cap)
        members, sizes, sums, cent, cent16, status = ops.bucket_table(cuda(g["keys"]), cuda(labels), pool,
                                                                       block // bucket, cap, want_bf16=True)
        assert np.array_equal(members.cpu().numpy(), want.bucket_members) and np.array_equal(members.cpu().numpy(), g["members"])
        assert np.array_equal(sizes.cpu().numpy(), want.bucket_sizes)
        assert np.array_equal(cent.cpu().numpy().view(np.int32), want.bucket_centroids.view(np.int32))
        assert torch.equal(cent16, cent.bfloat16()) and int(status) == 0
    from lsa_b200 import core
    members = core.members_from_labels(torch.tensor([1, 0, 1, 2, 0, 1]).cuda(), 3, 4)
    assert members.tolist() == [[1, 4, -1, -1], [0, 2, 5, -1], [3, -1, -1, -1]]


# ------------------------------------------------------------------------------------------------ selection


def _flat_case(T, d, pool, bucket, cap, block, seed, centres=24):
    raw = mixture(T, d, centres, 0.3, seed)
    keys = unit_rows(raw)
    rng = np.random.default_rng(seed + 1)
    return raw, keys, rng


@pytest.mark.parametrize("T,R,top_p,top_k,window,sink", [(4196, 300, 16, 2048, 512, 4), (40000, 257, 64, 700, 1024, 4),
                                                          (9000, 64, 200, 4096, 512, 0)])
def test_flat_read_is_bit_exact(ops, oracle, T, R, top_p, top_k, window, sink):
    raw, keys, rng = _flat_case(T, 64, 16, 64, 128, 512, T)
    buckets = oracle.build_buckets(keys, 16, 64, 128, 512)
    positions = np.sort(rng.integers(0, T, R))
    positions[:4] = [0, 1, 511, 512]
    queries = unit_rows(raw[positions] + 0.5 * rng.standard_normal((R, 64), dtype=np.float32))
    want_sel, want_len, want_picked, want_keys = oracle.read(queries, positions, buckets, top_p, top_k, sink, window,
                                                             return_picked=True)
    m = buckets.bucket_centroids.shape[0]
    visible = np.minimum(positions // 512 * 8, m).astype(np.int32)
    keys_out, picked = ops.flat_select(cuda(queries), cuda(buckets.bucket_centroids), cuda(visible), top_p)
    assert np.array_equal(keys_out.cpu().numpy(), want_keys)
    assert np.array_equal(picked.cpu().numpy(), want_picked)
    sel, lens, status = ops.expand(picked, cuda(positions), cuda(buckets.bucket_members), top_k, sink, window)
    assert np.array_equal(lens.cpu().numpy(), want_len) and np.array_equal(sel.cpu().numpy(), want_sel)
    assert int(status) == 0


def test_flat_read_golden_and_early_budget(oracle):
    from lsa_b200 import core
    from lsa_b200.budget import EarlyBudget
    g = golden("flat_small")
    buckets = core.Buckets(cuda(g["centroids"]), cuda(g["members"]), cuda(g["sizes"]), 8, 64)
    q, pos = cuda(g["queries"]), cuda(g["positions"])
    for tag, (top_p, top_k, window, early) in {"": (8, 48, 64, None), "_small": (3, 20, 16, None),
                                               "_early": (8, 48, 64, EarlyBudget(200, 12, 2))}.items():
        sel, lens = core.read(q, pos, buckets, top_p, top_k, 4, window, early_budget=early)
        assert np.array_equal(sel.cpu().numpy(), g["selected" + tag])
        assert np.array_equal(lens.cpu().numpy(), g["lengths" + tag])
    g = golden("flat_c1like")
    built = core.build_buckets(cuda(g["keys"]), 16, 64, 128, 512)
    assert np.array_equal(built.bucket_members.cpu().numpy(), g["members"])
    sel, lens = core.read(cuda(g["queries"]), cuda(g["positions"]), built, 16, 700, 4, 512)
    assert np.array_equal(sel.cpu().numpy(), g["selected_cut"]) and np.array_equal(lens.cpu().numpy(), g["lengths_cut"])


def test_selection_with_ties_rows_of_every_length_and_query_norms(ops, oracle):
    # thousands of identical centroids tie: the lower bucket wins, run to run the same
    rng = np.random.default_rng(5)
    base = unit_rows(rng.standard_normal((1, 64), dtype=np.float32))
    cents = np.repeat(base, 5000, axis=0)
    cents[::7] = unit_rows(rng.standard_normal((len(cents[::7]), 64), dtype=np.float32))
    queries = unit_rows(base + 0.01 * rng.standard_normal((40, 64), dtype=np.float32))
    queries[1] *= 0.01
    queries[2] *= 500.0
    visible = np.array([0, 1, 300, 1023, 2048, 2049, 4999, 5000] * 5, dtype=np.int32)
    want = np.full((40, 64), oracle.EMPTY_KEY, dtype=np.int64)
    for r in range(40):
        n = int(visible[r])
        keys = oracle.pack_keys(_dots(oracle, queries[r], cents[:n]), np.arange(n, dtype=np.int32))
        top = np.sort(keys)[::-1][:64]
        want[r, : len(top)] = top
    got, picked = ops.flat_select(cuda(queries), cuda(cents), cuda(visible), 64)
    again, _ = ops.flat_select(cuda(queries), cuda(cents), cuda(visible), 64)
    assert np.array_equal(got.cpu().numpy(), want) and torch.equal(got, again)
    assert np.array_equal(picked.cpu().numpy(), oracle.unpack_ids(want))


def _dots(oracle, query, rows):
    return oracle.scores(query, rows) if len(rows) else np.zeros(0, dtype=np.float32)


def test_decode_scan_and_candidate_merge(ops, oracle):
    rng = np.random.default_rng(9)
    lengths = [700, 2048, 5000, 64, 0, 33000]
    first = np.concatenate([[0], np.cumsum(lengths)[:-1]]).astype(np.int64)
    cents = unit_rows(rng.standard_normal((sum(lengths), 64), dtype=np.float32))
    queries = unit_rows(rng.standard_normal((len(lengths), 64), dtype=np.float32))
    want = np.full((len(lengths), 32), oracle.EMPTY_KEY, dtype=np.int64)
    for r, n in enumerate(lengths):
        keys = oracle.pack_keys(_dots(oracle, queries[r], cents[first[r]: first[r] + n]), np.arange(n, dtype=np.int32))
        top = np.sort(keys)[::-1][:32]
        want[r, : len(top)] = top
    for splits in (1, 4, 37):
        got, picked = ops.flat_select_decode(cuda(queries), cuda(cents), cuda(first), cuda(np.array(lengths, np.int32)),
                                             32, splits)
        assert np.array_equal(got.cpu().numpy(), want), splits
        assert np.array_equal(picked.cpu().numpy(), oracle.unpack_ids(want))
    # merging lists that several owners of disjoint bucket ranges produced gives the global list
    parts = []
    for lo, hi in ((0, 11000), (11000, 22000), (22000, 33000)):
        k = oracle.pack_keys(_dots(oracle, queries[5], cents[first[5] + lo: first[5] + hi]), np.arange(lo, hi, dtype=np.int32))
        parts.append(np.sort(k)[::-1][:32])
    merged, ids = ops.merge_candidates(cuda(np.stack(parts)[:, None, :]))
    assert np.array_equal(merged.cpu().numpy()[0], want[5])


def test_beam_step_matches_the_oracle_tree_read(ops, oracle):
    g = golden("hierarchy")
    q = cuda(g["queries"])
    R = q.shape[0]
    nodes, kids = cuda(g["node_centroids_0"]), cuda(g["children_0"])
    # level 1 scored whole, the best 3 kept and their children carried to the buckets
    zero = torch.zeros(R, dtype=torch.int32).cuda()
    end = torch.full((R,), nodes.shape[0], dtype=torch.int32).cuda()
    kept, keys = ops.beam_step(q, nodes, None, zero, end, 3)
    carried = ops.beam_step(q, nodes, None, zero, end, 3, children=kids)
    scores = g["queries"] @ g["node_centroids_0"].T
    for r in range(R):
        order = np.argsort(-scores[r], kind="stable")[:3]
        assert set(kept[r].tolist()) == set(order.tolist())
        assert carried[r].tolist() == g["children_0"][kept[r].cpu().numpy()].reshape(-1).tolist()
    # level 0: carried children beside a run of uncovered buckets, top 16
    first = torch.full((R,), 1000, dtype=torch.int32).cuda()
    last = torch.full((R,), 1024, dtype=torch.int32).cuda()
    picked, _ = ops.beam_step(q, cuda(g["centroids"]), carried, first, last, 16)
    for r in range(R):
        cand = np.concatenate([carried[r].cpu().numpy(), np.arange(1000, 1024)])
        keys = oracle.pack_keys(_dots(oracle, g["queries"][r], g["centroids"])[cand], cand.astype(np.int32))
        want = oracle.unpack_ids(np.sort(keys)[::-1][:16])
        assert picked[r].tolist() == want.tolist()


# ------------------------------------------------------------------------------------------------ expansion


def test_expansion_with_slots_owners_and_bad_ids(ops, oracle):
    g = golden("flat_c1like")
    buckets = oracle.Buckets(g["centroids"], g["members"], g["sizes"], 8, 512)
    _, _, picked, _ = oracle.read(g["queries"], g["positions"], buckets, 16, 700, 4, 512, return_picked=True)
    pos, mem = cuda(g["positions"]), cuda(g["members"])
    want_sel, want_len = oracle.expand(picked, g["positions"], g["members"], 700, 4, 512)
    # KV slots through a permuted page table
    rng = np.random.default_rng(2)
    pages = rng.permutation(70).astype(np.int32)
    sel, lens, _ = ops.expand(cuda(picked), pos, mem, 700, 4, 512, page_table=cuda(pages), page_size=64)
    mapped = np.where(want_sel >= 0, pages[np.maximum(want_sel, 0) // 64] * 64 + np.maximum(want_sel, 0) % 64, -1)
    assert np.array_equal(sel.cpu().numpy(), mapped) and np.array_equal(lens.cpu().numpy(), want_len)
    # two owners of halves of the sequence hold the whole list between them, each id once
    lo, _, _ = ops.expand(cuda(picked), pos, mem, 700, 4, 512, owner=(0, 2048))
    hi, _, _ = ops.expand(cuda(picked), pos, mem, 700, 4, 512, owner=(2048, 1 << 40))
    for a, b, w in zip(lo.cpu().numpy(), hi.cpu().numpy(), want_sel):
        assert sorted(a[a >= 0].tolist() + b[b >= 0].tolist()) == sorted(w[w >= 0].tolist())
        assert (a[a >= 0] < 2048).all() and (b[b >= 0] >= 2048).all()
    # four ranks that hold the cache dealt out in granules of 64 positions: each writes rows of its own share
    seen = [[] for _ in want_sel]
    for rank in range(4):
        part, lens_r, _ = ops.expand(cuda(picked), pos, mem, 700, 4, 512, dealt=(64, 4, rank))
        for r, row in enumerate(part.cpu().numpy()):
            local = row[row >= 0]
            assert len(local) == int(lens_r[r])
            seen[r] += (local // 64 * 256 + rank * 64 + local % 64).tolist()
    for got, w in zip(seen, want_sel):
        assert sorted(got) == sorted(w[w >= 0].tolist())
    # a pick past the table is counted in the status word and skipped
    bad = picked.copy()
    bad[0, 0] = 10**6
    _, _, status = ops.expand(cuda(bad), pos, mem, 700, 4, 512)
    assert int(status) == 1


def test_expansion_of_decode_rows_by_a_cluster(ops, oracle):
    """Eight rows or fewer whose picks hold tens of thousands of ids (a decode step over a long context) go through
    the kernel that gives a row a cluster of CTAs; its lists are the oracle's, id for id: full picks, picks that are
    fewer than the cluster's CTAs, a cut at top_k inside a bucket, holes in the picks, per-row budgets, a page
    table, the window and sinks left out."""
    rng = np.random.default_rng(4)
    cap, buckets_n, T = 1024, 300, 300 * 1024 + 5000
    members = np.full((buckets_n, cap), -1, dtype=np.int32)
    for b in range(buckets_n):  # pools of 64 consecutive positions, 6 to 16 a bucket, ascending
        pools = np.sort(rng.choice(np.arange(b * 16, b * 16 + 16), int(rng.integers(6, 17)), replace=False))
        ids = (pools[:, None] * 64 + np.arange(64)[None]).reshape(-1)
        members[b, : len(ids)] = ids
    positions = np.array([T - 1, T - 700, 200000, 70, 5000], dtype=np.int64)
    for top_p, top_k in ((40, 40 * cap), (40, 9000), (5, 5 * cap + 30000)):
        picked = np.stack([rng.choice(buckets_n, top_p, replace=False) for _ in positions]).astype(np.int32)
        picked[1, 3] = -1
        picked[2, :] = np.sort(picked[2])
        if top_p > 8:
            picked[3, 0] = 0  # the bucket of the sinks, for a row whose window starts at 0
        want_sel, want_len = oracle.expand(picked, positions, members, top_k, 4, 2048)
        sel, lens, _ = ops.expand(cuda(picked), cuda(positions), cuda(members), top_k, 4, 2048)
        assert np.array_equal(lens.cpu().numpy(), want_len), (top_p, top_k)
        assert np.array_equal(sel.cpu().numpy(), want_sel), (top_p, top_k)
    row_p = np.array([40, 7, 40, 1, 12], dtype=np.int32)
    row_k = np.array([40 * cap, 3000, 100, 40 * cap, 5000], dtype=np.int32)
    pages = rng.permutation(T // 64 + 1).astype(np.int32)
    sel, lens, _ = ops.expand(cuda(picked), cuda(positions), cuda(members), 40 * cap, 4, 2048, cuda(row_p), cuda(row_k),
                              page_table=cuda(pages), page_size=64, local=False)
    one, one_len, _ = ops.expand(cuda(picked), cuda(positions), cuda(members), 40 * cap, 4, 2048, cuda(row_p),
                                 cuda(row_k), page_table=cuda(pages), page_size=64, local=False, owner=(0, 1 << 40))
    assert torch.equal(lens, one_len)  # (an owner range takes the one-warp kernel)
    for r in range(len(positions)):
        assert torch.equal(sel[r, : int(lens[r])], one[r, : int(lens[r])])


def test_expansion_of_a_few_rows_with_long_lists(ops, oracle):
    """Up to 64 rows whose picks hold over a thousand ids go through the CTA-a-row kernel; its lists are the
    one-warp kernel's and the oracle's, id for id - cut at top_k, under per-row budgets, through a page table."""
    g = golden("flat_c1like")
    buckets = oracle.Buckets(g["centroids"], g["members"], g["sizes"], 8, 512)
    rows = slice(40, 88)
    positions = g["positions"][rows]
    _, _, picked, _ = oracle.read(g["queries"][rows], positions, buckets, 16, 700, 4, 512, return_picked=True)
    pos, mem = cuda(positions), cuda(g["members"])
    for top_k in (700, 150, 4000):
        want_sel, want_len = oracle.expand(picked, positions, g["members"], top_k, 4, 512)
        sel, lens, _ = ops.expand(cuda(picked), pos, mem, top_k, 4, 512)
        assert np.array_equal(sel.cpu().numpy(), want_sel) and np.array_equal(lens.cpu().numpy(), want_len), top_k
    # the early budget of the first rows
    cut = int(positions[20])
    want_sel, want_len = oracle.expand(picked, positions, g["members"], 700, 4, 512, early_budget=(cut, 90, 5))
    early = positions < cut
    row_p = cuda(np.where(early, 5, 16).astype(np.int32))
    row_k = cuda(np.where(early, 90, 700).astype(np.int32))
    sel, lens, _ = ops.expand(cuda(picked), pos, mem, 700, 4, 512, row_p, row_k)
    assert np.array_equal(sel.cpu().numpy(), want_sel) and np.array_equal(lens.cpu().numpy(), want_len)
    # KV slots through a page table, the window and sinks left out, a pick past the table
    pages = np.random.default_rng(3).permutation(70).astype(np.int32)
    want_sel, want_len = oracle.expand(picked, positions, g["members"], 700, 4, 512)
    sel, lens, _ = ops.expand(cuda(picked), pos, mem, 700, 4, 512, page_table=cuda(pages), page_size=64)
    mapped = np.where(want_sel >= 0, pages[np.maximum(want_sel, 0) // 64] * 64 + np.maximum(want_sel, 0) % 64, -1)
    assert np.array_equal(sel.cpu().numpy(), mapped) and np.array_equal(lens.cpu().numpy(), want_len)
    bare, bare_len, _ = ops.expand(cuda(picked), pos, mem, 700, 4, 512, local=False)
    for r in range(len(positions)):
        n = int(bare_len[r])
        assert np.array_equal(bare[r, :n].cpu().numpy(), want_sel[r, :n]) and (bare[r, n:] == -1).all()
        assert n == int(want_len[r]) - min(512, int(positions[r]) + 1) - min(4, max(0, int(positions[r]) + 1 - 512))
    bad = picked.copy()
    bad[3, 1] = 10**6
    sel, _, status = ops.expand(cuda(bad), pos, mem, 700, 4, 512)
    assert int(status) == 1
    keep = np.delete(bad[3], 1)[None]
    want_row, _ = oracle.expand(np.concatenate([keep, np.full((1, 1), -1, np.int32)], 1), positions[3:4],
                                g["members"], 700, 4, 512)
    assert np.array_equal(sel[3].cpu().numpy(), want_row[0])


# ------------------------------------------------------------------------------------------------ attention


def _attend_case(T, Hq, Hkv, dh, R, L, seed):
    q, k, v = layer_inputs(T, Hq, Hkv, dh, 16, seed)
    rng = np.random.default_rng(seed)
    rows = np.sort(rng.choice(T, R, replace=False))
    ids = np.full((R, L), -1, dtype=np.int32)
    lens = np.zeros(R, dtype=np.int32)
    for i, pos in enumerate(rows):
        n = min(L, pos + 1, int(rng.integers(0, L + 1)))
        ids[i, :n] = rng.choice(pos + 1, n, replace=False)
        lens[i] = n
    return q, k, v, rows, ids, lens


@pytest.mark.parametrize("T,Hq,Hkv,dh,R,L,splits", [(3000, 40, 8, 128, 24, 700, 1), (3000, 8, 2, 128, 40, 333, 1),
                                                    (2000, 16, 1, 64, 16, 500, 1), (5000, 40, 8, 128, 6, 3000, 5),
                                                    (1500, 4, 4, 64, 10, 100, 3)])
def test_sparse_attention_within_bf16_tolerance(ops, oracle, T, Hq, Hkv, dh, R, L, splits):
    q, k, v, rows, ids, lens = _attend_case(T, Hq, Hkv, dh, R, L, T + L)
    lens[0] = 0  # a row that reads nothing
    scale = dh ** -0.5
    want, want_lse = oracle.sparse_attend(q[rows], k, v, ids, rows, 0, 0, scale, lengths=lens)
    out, lse = ops.sparse_attend(cuda(q[rows], torch.bfloat16), cuda(k, torch.bfloat16), cuda(v, torch.bfloat16),
                                 cuda(ids), cuda(lens), scale, splits=splits, out_dtype=torch.float32)
    err = np.abs(out.cpu().numpy() - want)
    assert err.max() <= 2e-2 and err.mean() <= 2e-3, (err.max(), err.mean())
    got_lse = lse.cpu().numpy()
    assert np.isneginf(got_lse[0]).all() and not out[0].any()
    np.testing.assert_allclose(got_lse[1:], want_lse[1:], rtol=0, atol=2e-3)
    out16, _ = ops.sparse_attend(cuda(q[rows], torch.bfloat16), cuda(k, torch.bfloat16), cuda(v, torch.bfloat16),
                                 cuda(ids), cuda(lens), scale, splits=splits)
    assert np.abs(out16.float().cpu().numpy() - want).max() <= 2e-2


@pytest.mark.parametrize("T,Hq,Hkv,dh,first", [(40, 4, 2, 64, 0), (300, 8, 1, 128, 0), (131, 6, 2, 128, 260)])
def test_a_value_that_is_not_finite_reaches_the_rows_that_read_it(ops, T, Hq, Hkv, dh, first):
    """Dense causal rows of both forms, in bf16 and fp32, to tensors that start anywhere: the gather's rows are not numbers, and
    the rows before it are what they are without the value."""
    n = first + T
    q, k, v = (cuda(x, torch.bfloat16) for x in layer_inputs(n, Hq, Hkv, dh, 16, n))
    q = q[first:]
    ids = torch.arange(n, device="cuda", dtype=torch.int32).expand(T, n).contiguous()
    lengths = first + 1 + torch.arange(T, device="cuda", dtype=torch.int32)
    clean = ops.causal_attend(q, k, v, first, dh ** -0.5, out=torch.empty(T, Hq, dh, device="cuda"))
    for x, at, what in ((v, first + 20, float("nan")), (v, n - 1, float("inf")), (k, first + 9, float("nan")), (k, n - 2, float("-inf"))):
        kept = x[at, 0, 3].clone()
        x[at, 0, 3] = what
        want, _ = ops.sparse_attend(q, k, v, ids, lengths, dh ** -0.5)
        room = torch.empty(q.numel() + 1, device="cuda", dtype=torch.bfloat16)
        for out in (room[1:].view(T, Hq, dh), room[:-1].view(T, Hq, dh), torch.empty(T, Hq, dh, device="cuda")):
            got = ops.causal_attend(q, k, v, first, dh ** -0.5, out=out)
            assert torch.equal(got.isnan(), want.isnan()) and torch.equal(got.isinf(), want.isinf())
            same = want.isfinite()
            assert (got.float() - want.float())[same].abs().max() <= 2e-2 and not same.all()
            before = clean[:at - first]  # (read again in fp32 where the tile holds the value: one rounding to bf16 apart)
            assert ((got[:at - first].float() - before).abs() <= 2 ** -8 * before.abs() + 2 ** -13).all()
        x[at, 0, 3] = kept


@pytest.mark.parametrize("T,Hq,Hkv,dh", [(90, 8, 2, 64), (127, 16, 1, 128), (128, 8, 2, 128), (300, 5, 1, 64), (1153, 16, 2, 128)])
def test_a_dense_read_is_as_close_to_64_bits_as_the_gather_of_every_key(ops, T, Hq, Hkv, dh):
    """Causal rows over clustered keys, probabilities as two bf16 terms, both forms. Two terms leave 2^-17 of a probability;
    exponents of up to 32 in fp32 are off by 2^-19 of it and the sums by less: 2^-16 in all."""
    q, k, v = (cuda(x, torch.bfloat16) for x in layer_inputs(T, Hq, Hkv, dh, 16, T))
    ids = torch.arange(T, device="cuda", dtype=torch.int32).expand(T, T).contiguous()
    gather, _ = ops.sparse_attend(q, k, v, ids, 1 + ids[0], dh ** -0.5, out_dtype=torch.float32)
    scores = torch.einsum("qhd,khd->hqk", q.double(), k.double().repeat_interleave(Hq // Hkv, dim=1)) * dh ** -0.5
    scores.masked_fill_(torch.ones(T, T, device="cuda").triu(1).bool(), -float("inf"))
    want = torch.einsum("hqk,khd->qhd", scores.softmax(-1), v.double().repeat_interleave(Hq // Hkv, dim=1))
    far = lambda got: float((got.double() - want).norm() / want.norm())
    for warp_mma in (False, True):
        out, lse = ops.band_attend(q, k, v, 0, T, 0, dh ** -0.5, warp_mma=warp_mma, two_term=True)
        assert far(out) <= min(2 ** -16, far(gather)), (far(out), far(gather))
        assert (lse - scores.logsumexp(-1).t()).abs().max() <= 1e-4


@pytest.mark.parametrize("T,Hq,Hkv,dh,window,sink,first,R", [(3000, 40, 8, 128, 1024, 4, 1500, 700),
                                                             (700, 8, 2, 128, 512, 4, 0, 700),
                                                             (2000, 16, 1, 64, 300, 0, 90, 333),
                                                             (2500, 8, 8, 64, 64, 7, 1000, 61)])
def test_band_attention_and_its_hand_over_to_the_gather(ops, oracle, T, Hq, Hkv, dh, window, sink, first, R):
    q, k, v = layer_inputs(T, Hq, Hkv, dh, 16, T + window)
    rows = np.arange(first, first + R)
    scale = dh ** -0.5
    empty = np.full((R, 1), -1, dtype=np.int32)
    want, want_lse = oracle.sparse_attend(q[rows], k, v, empty, rows, window, sink, scale)
    Q, K, V = cuda(q[rows], torch.bfloat16), cuda(k, torch.bfloat16), cuda(v, torch.bfloat16)
    # both forms: tensor memory (dense heads of 128 dims, 128 rows or more) and warp-level tiles
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    for warp_mma in (True, False):
        out, lse = ops.band_attend(Q, K, V, first, window, sink, scale, warp_mma=warp_mma, status=status)
        err = np.abs(out.cpu().numpy() - want)
        assert err.max() <= 2e-2 and err.mean() <= 2e-3, (warp_mma, err.max(), err.mean())
        np.testing.assert_allclose(lse.cpu().numpy(), want_lse, rtol=0, atol=2e-3)
    assert int(status) == 0
    # the gather continues from the band's partial result over keys outside the window and the sinks
    rng = np.random.default_rng(1)
    ids = np.full((R, 200), -1, dtype=np.int32)
    lens = np.zeros(R, dtype=np.int32)
    for i, pos in enumerate(rows):
        lo, hi = sink, max(sink, pos + 1 - window)
        n = min(200, hi - lo)
        if n > 0:
            ids[i, :n] = rng.choice(np.arange(lo, hi), n, replace=False)
        lens[i] = max(n, 0)
    whole, whole_lse = oracle.sparse_attend(q[rows], k, v, ids, rows, window, sink, scale, lengths=lens)
    for splits in (1, 3):
        got, got_lse = ops.sparse_attend(Q, K, V, cuda(ids), cuda(lens), scale, splits=splits, out_dtype=torch.float32,
                                         init=(out, lse))
        err = np.abs(got.cpu().numpy() - whole)
        assert err.max() <= 2e-2 and err.mean() <= 2e-3, (splits, err.max(), err.mean())
        np.testing.assert_allclose(got_lse.cpu().numpy(), whole_lse, rtol=0, atol=2e-3)


def test_attention_skips_bad_ids_and_merges_partials(ops, oracle):
    q, k, v, rows, ids, lens = _attend_case(2000, 8, 2, 128, 12, 400, 4)
    scale = 128 ** -0.5
    want, want_lse = oracle.sparse_attend(q[rows], k, v, ids, rows, 0, 0, scale, lengths=lens)
    spoiled = ids.copy()
    spoiled = np.concatenate([spoiled, np.full((12, 8), 10**7, np.int32)], axis=1)
    for r in range(12):  # ids past the cache and negative ids inside the list are skipped
        spoiled[r, lens[r]: lens[r] + 4] = [-5, 10**7, -1, 2000]
    Q, K, V = cuda(q[rows], torch.bfloat16), cuda(k, torch.bfloat16), cuda(v, torch.bfloat16)
    out, lse = ops.sparse_attend(Q, K, V, cuda(spoiled), cuda(lens + 4), scale, out_dtype=torch.float32)
    assert np.abs(out.cpu().numpy() - want).max() <= 2e-2
    # halves of every list attended apart, merged by their log-sum-exps
    a = np.where(np.arange(400)[None, :] % 2 == 0, ids, -1)
    b = np.where(np.arange(400)[None, :] % 2 == 1, ids, -1)
    oa, la = ops.sparse_attend(Q, K, V, cuda(a), cuda(lens), scale, out_dtype=torch.float32)
    ob, lb = ops.sparse_attend(Q, K, V, cuda(b), cuda(lens), scale, out_dtype=torch.float32)
    merged, mlse = ops.lse_merge(torch.stack([oa, ob]), torch.stack([la, lb]))
    assert np.abs(merged.cpu().numpy() - want).max() <= 2e-2
    ok = np.isfinite(want_lse)
    np.testing.assert_allclose(mlse.cpu().numpy()[ok], want_lse[ok], rtol=0, atol=2e-3)
    cpu_merge, _ = oracle.lse_merge(torch.stack([oa, ob]).cpu().numpy(), torch.stack([la, lb]).cpu().numpy())
    np.testing.assert_allclose(merged.cpu().numpy(), cpu_merge, rtol=0, atol=1e-5)


def test_topk_attention_reproduces_the_reference(oracle):
    from lsa_b200 import core
    g = golden("attention")
    q, k, v = (cuda(bf16_round(g[n]))[None] for n in "qkv")
    T, dh = g["q"].shape[0], g["q"].shape[2]
    # dh 16 is below what the tensor-core kernel takes: the call is refused, not rerouted
    with pytest.raises(ValueError, match="shape outside"):
        core.topk_attention(q, k, v, cuda(g["selected"])[None], 8, 2, dh ** -0.5)
    m = golden("mini_c1")
    bf = lambda bits: (torch.from_numpy(bits.astype(np.int32)) << 16).view(torch.float32)
    Q, K, V = bf(m["q_bf16"]).cuda(), bf(m["k_bf16"]).cuda(), bf(m["v_bf16"]).cuda()
    out = core.topk_attention(Q[None], K[None], V[None], cuda(m["selected"])[None], 128, 4, 64 ** -0.5)
    err = np.abs(out[0].cpu().numpy()[m["out_rows"]] - m["out"])
    assert err.max() <= 2e-2 and err.mean() <= 2e-3
    # full budget is dense causal attention; future keys in the selection are dropped
    full = torch.arange(1024, dtype=torch.int32).expand(1, 1024, 1024).contiguous().cuda()
    dense = core.topk_attention(Q[None], K[None], V[None], full, 0, 0, 64 ** -0.5)
    window = core.topk_attention(Q[None], K[None], V[None], torch.full((1, 1024, 1), -1, dtype=torch.int32).cuda(),
                                 1024, 0, 64 ** -0.5)
    assert (dense - window).abs().max() <= 2e-2


def test_cpu_tensors_are_refused(ops):
    with pytest.raises(RuntimeError, match="no CPU path"):
        ops.pool_keys(torch.zeros(1, 16, 8), 4)


def test_few_row_paths_of_a_decode_step(ops, oracle):
    """The buckets a position sees against torch's; a few rows' scan split over CTAs against the chunk's scan, key for key;
    the few-row map's vector loads against its plain ones, bit for bit; merges of up to 33 parts against 64-bit sums."""
    gen = torch.Generator(device="cuda").manual_seed(2)
    positions = torch.tensor([0, 1, 1023, 1024, 5000, 1 << 40], device="cuda")
    for block, per, limit in ((1024, 32, 100), (64, 8, 1 << 30), (1, 1, 0)):
        want = (positions // block * per).clamp_max(limit).to(torch.int32)
        assert torch.equal(ops.visible_buckets(positions, block, per, limit), want)
    for d, m in ((64, 1), (64, 1024), (64, 1025), (32, 5000)):
        rows = torch.nn.functional.normalize(torch.randn(8, d, generator=gen, device="cuda"), dim=1)
        cent = torch.nn.functional.normalize(torch.randn(m, d, generator=gen, device="cuda"), dim=1)
        visible = torch.randint(0, m + 1, (8,), generator=gen, device="cuda", dtype=torch.int32)
        visible[0] = m
        for keep in (1, 64, 128):
            want, _ = ops.flat_select(rows, cent, visible, keep)
            got, _ = ops.flat_select_decode(rows, cent, None, visible, keep, splits=1 if m <= 1024 else -(-m // 512))
            assert torch.equal(got, want)
    x = torch.randn(5, 10, 128, generator=gen, device="cuda").bfloat16()
    for cols in (64, 128):
        w = torch.randn(256, cols, generator=gen, device="cuda").bfloat16()
        shifted = torch.empty(256 * cols + 1, device="cuda", dtype=torch.bfloat16)[1:].view(256, cols).copy_(w)
        got, plain = ops.index_map(x, w, group=5), ops.index_map(x, shifted, group=5)
        assert torch.equal(got, plain) and shifted.data_ptr() % 16 != 0
        want = torch.nn.functional.normalize(x.double().view(5, 2, 5, 128).sum(2).view(5, 256) @ w.double(), dim=1)
        assert (got.double() - want).abs().max() <= 1e-5  # (256 fp32 terms in eight partial sums, unit rows)
    for n in (1, 2, 15, 16, 17, 32, 33):
        for dh in (8, 128, 264):
            parts = torch.randn(n, 1030, dh, generator=gen, device="cuda")
            lses = 3 * torch.randn(n, 1030, generator=gen, device="cuda")
            lses[0, 5], lses[:, 6] = -float("inf"), -float("inf")
            out, lse = ops.lse_merge(parts, lses)
            weights = torch.softmax(lses.double(), 0).nan_to_num(0.0)
            assert (out.double() - (weights[..., None] * parts.double()).sum(0)).abs().max() <= 1e-5
            assert (lse - torch.logsumexp(lses.double(), 0))[torch.isfinite(lse)].abs().max() <= 1e-5
            assert not torch.isfinite(lse[6]) and not out[6].any()


@pytest.mark.parametrize("kernel", ["gather", "scan", "decode scan", "merge", "ward", "bucket table", "map", "row map"])
def test_host_threads_that_launch_a_kernel_with_different_sizes(ops, kernel, monkeypatch):
    """The library lets go of the interpreter's lock, so a decode step's small launch and a chunk's large one of the same
    kernel meet: neither may have the other refused. (The outputs are those of a call alone.)"""
    from lsa_b200 import _lib

    gen = torch.Generator(device="cuda").manual_seed(3)
    rand = lambda *shape: torch.randn(*shape, generator=gen, device="cuda")
    if kernel == "gather":
        q, k = rand(2000, 8, 128).bfloat16(), rand(64, 2, 128).bfloat16()
        ids = torch.arange(8, device="cuda", dtype=torch.int32).expand(2000, 8).contiguous()
        run = lambda big: ops.sparse_attend(q if big else q[:1], k, k, ids if big else ids[:1], None, 0.1)[0]
    elif kernel in ("scan", "decode scan"):
        rows, cent, seen = rand(16, 64), rand(700, 64), torch.full((16,), 700, device="cuda", dtype=torch.int32)
        scan = ops.flat_select if kernel == "scan" else lambda r, c, s, top: ops.flat_select_decode(r, c, None, s, top)
        run = lambda big: scan(rows, cent, seen, 512 if big else 1)[0]
    elif kernel == "merge":
        keys = {n: torch.randint(0, 1 << 60, (n, 4, 256), generator=gen, device="cuda") for n in (2, 32)}
        run = lambda big: ops.merge_candidates(keys[32 if big else 2])[0]
    elif kernel == "ward":
        pools = torch.nn.functional.normalize(rand(1, 512, 64), dim=2)
        run = lambda big: ops.ward_rounds(pools if big else pools[:, :8].contiguous(), 1.0, 64 if big else 4, 16.0)[0]
    elif kernel == "bucket table":
        keys, labels = rand(600 * 32, 64), torch.arange(600 * 32, device="cuda").view(600, 32) % 16
        run = lambda big: ops.bucket_table(keys if big else keys[:32], labels if big else labels[:1], 1, 16, 4)[2]
    elif kernel == "map":
        x, w = rand(100, 2, 64), {n: rand(128, n) for n in (8, 64)}
        run = lambda big: ops.index_map(x, w[64 if big else 8], group=1)
    else:
        x, w = rand(8, 2, 512).bfloat16(), rand(64, 1024).bfloat16()
        run = lambda big: ops.rows_linear(x if big else x[:1], w)
    entries = {}  # the entry point and the arguments of each call, to be made again with nothing in between

    def recorded(name, *args, launches=1):
        entries[len(entries)] = getattr(_lib.load(), name), args
        return _lib.call(name, *args, launches=launches)

    monkeypatch.setattr(ops, "call", recorded)
    outs = [run(False), run(True)]
    torch.cuda.synchronize()
    want, wrong = [out.clone() for out in outs], []

    def work(which):
        entry, args = entries[which]
        wrong.extend(code for code in (entry(*args) for _ in range(4000)) if code != 0)

    threads = [threading.Thread(target=work, args=(which,)) for which in (0, 1, 0, 1)]
    for thread in threads:
        thread.start()
    for thread in threads:
        thread.join()
    assert len(entries) == 2 and not wrong, (len(entries), wrong[:3])
    assert all(torch.equal(out, same) for out, same in zip(outs, want))


@pytest.mark.parametrize("n,d", [(1, 1), (5, 64), (70001, 64), (3000, 20), (17, 200), (4, 30)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_unit_rows_in_one_pass_are_the_check_s(ops, n, d, dtype):
    """The greatest distance from unit length against 64 bits (fp32 sums of up to 200 squares: 2e-6), what is not finite, and the
    check's errors from either form."""
    from lsa_b200 import core

    gen = torch.Generator(device="cuda").manual_seed(n + d)
    rows = torch.nn.functional.normalize(torch.randn(n, d, device="cuda", generator=gen), dim=-1).to(dtype)
    rows[n // 2] *= 0.75
    finite, off = ops.unit_rows(rows).tolist()
    assert finite == 1.0 and abs(off - float((rows.double().norm(dim=1) - 1).abs().max())) <= 2e-6
    apart = torch.empty(n, d + 1, device="cuda", dtype=dtype)[:, 1:].copy_(rows)
    for x in (rows, apart):
        with pytest.raises(ValueError, match="unit rows - a row is 0.2"):
            core.check_unit_rows("rows", x)
        for bad in (float("nan"), float("inf"), -float("inf")):
            worse = x.clone()
            worse[n - 1, d - 1] = bad
            with pytest.raises(ValueError, match="non-finite"):
                core.check_unit_rows("rows", worse)
    core.check_unit_rows("rows", torch.nn.functional.normalize(rows.float(), dim=-1))
    with pytest.raises(ValueError, match="unit rows"):
        core.check_unit_rows("rows", torch.full((2, 8), 1e30, device="cuda"))
    unaligned = torch.empty(n * d + 1, device="cuda", dtype=dtype)[1:].view(n, d).copy_(rows)
    assert torch.equal(ops.unit_rows(unaligned)[0], torch.ones((), device="cuda")) and abs(float(ops.unit_rows(unaligned)[1]) - off) <= 2e-6
