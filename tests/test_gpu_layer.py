"""One flat layer end to end on the GPU against the oracle: config 1's shapes cut to a few thousand tokens, the
served GQA shapes, and decode rows against their prefill rows."""

import numpy as np
import pytest
import torch

from helpers import bf16_round, cuda, layer_inputs

pytestmark = pytest.mark.gpu


def _layer(Hq, Hkv, dh, d_idx, design, seed):
    from lsa_b200.layer import FlatLayer

    rng = np.random.default_rng(seed)
    w = bf16_round(rng.standard_normal((2, Hkv * dh, d_idx), dtype=np.float32) / np.sqrt(Hkv * dh))
    return FlatLayer(design, cuda(w[0], torch.bfloat16), cuda(w[1], torch.bfloat16), Hq, Hkv, dh), w


@pytest.mark.parametrize("T,Hq,Hkv,dh,d_idx,sizes", [
    (4096 + 200, 8, 2, 128, 32, dict(pool_size=16, bucket_size=64, bucket_cap=128, cluster_block_size=512, top_p=4,
                                     top_k=512, sink_size=4, window_size=512)),
    (6144, 40, 8, 128, 64, dict(pool_size=16, bucket_size=32, bucket_cap=64, cluster_block_size=1024, top_p=16,
                                top_k=1024, sink_size=4, window_size=1024)),
])
def test_prefill_matches_the_oracle_stage_by_stage(oracle, T, Hq, Hkv, dh, d_idx, sizes):
    from lsa_b200.layer import FlatDesign

    design = FlatDesign(**sizes)
    layer, w = _layer(Hq, Hkv, dh, d_idx, design, T)
    q, k, v = layer_inputs(T, Hq, Hkv, dh, 32, T + 1)
    Q, K, V = (cuda(a, torch.bfloat16) for a in (q, k, v))
    out, index = layer.prefill(Q, K, V, chunk=2048, return_index=True)
    # index vectors: float, within rounding of the fixed-order oracle
    want_q = oracle.project(oracle.regroup_queries(q, Hkv), w[0])
    want_k = oracle.project(k.reshape(T, -1), w[1])
    index_q = layer.index_queries(Q).cpu().numpy()
    index_k = index.index_keys.cpu().numpy()
    # (tensor-core accumulation order differs from the oracle's: a few 1e-6 on unit rows)
    assert np.abs(index_q - want_q).max() < 3e-5 and np.abs(index_k - want_k).max() < 3e-5
    # from the device's own index vectors on, every integer result is the oracle's
    buckets = oracle.build_buckets(index_k, design.pool_size, design.bucket_size, design.bucket_cap,
                                   design.cluster_block_size)
    assert np.array_equal(index.buckets.bucket_members.cpu().numpy(), buckets.bucket_members)
    assert np.array_equal(index.buckets.bucket_centroids.cpu().numpy().view(np.int32),
                          buckets.bucket_centroids.view(np.int32))
    positions = np.arange(T)
    lists, lengths = layer.select(cuda(index_q), cuda(positions), index)
    want_lists, want_lengths = oracle.read(index_q, positions, buckets, design.top_p, design.top_k, design.sink_size,
                                           design.window_size)
    assert np.array_equal(lengths.cpu().numpy(), want_lengths)
    assert np.array_equal(lists.cpu().numpy(), want_lists)
    # and against the oracle's own index vectors the selection is the same except where two scores nearly tie
    own = oracle.build_buckets(want_k, design.pool_size, design.bucket_size, design.bucket_cap,
                               design.cluster_block_size)
    own_lists, _ = oracle.read(want_q, positions, own, design.top_p, design.top_k, design.sink_size,
                               design.window_size)
    same = np.mean([np.array_equal(a, b) for a, b in zip(own_lists, want_lists)])
    assert same >= 0.98, same
    rows = np.arange(0, T, 37)
    want, _ = oracle.sparse_attend(q[rows], k, v, want_lists[rows], rows, 0, 0, dh ** -0.5, lengths=want_lengths[rows])
    err = np.abs(out.float().cpu().numpy()[rows] - want)
    assert err.max() <= 2e-2 and err.mean() <= 2e-3, (err.max(), err.mean())


def test_a_decode_step_matches_its_prefill_row(oracle):
    from lsa_b200.layer import FlatDesign

    design = FlatDesign(pool_size=4, bucket_size=16, bucket_cap=32, cluster_block_size=256, top_p=8, top_k=256,
                        sink_size=4, window_size=256)
    T, Hq, Hkv, dh = 3000, 40, 8, 128
    layer, _ = _layer(Hq, Hkv, dh, 64, design, 3)
    q, k, v = layer_inputs(T, Hq, Hkv, dh, 16, 4)
    Q, K, V = (cuda(a, torch.bfloat16) for a in (q, k, v))
    out, index = layer.prefill(Q, K, V, chunk=1024, return_index=True)
    rows = torch.tensor([5, 255, 256, 1000, 2999]).cuda()
    for splits in (1, 4):
        step = layer.decode(Q[rows], rows, K, V, index, splits=splits)
        assert (step.float() - out[rows].float()).abs().max() <= 1e-2


def test_prefill_from_pinned_host_memory_is_the_resident_prefill():
    from lsa_b200.layer import FlatDesign

    design = FlatDesign(pool_size=16, bucket_size=32, bucket_cap=64, cluster_block_size=1024, top_p=16, top_k=1024,
                        sink_size=4, window_size=1024)
    T, Hq, Hkv, dh = 6144 + 300, 40, 8, 128
    layer, _ = _layer(Hq, Hkv, dh, 64, design, 9)
    q, k, v = (torch.from_numpy(a).bfloat16().pin_memory() for a in layer_inputs(T, Hq, Hkv, dh, 32, 10))
    want = layer.prefill(q.cuda(), k.cuda(), v.cuda(), chunk=2048)
    out = torch.empty(T, Hq, dh, dtype=torch.bfloat16).pin_memory()
    for _ in range(2):  # the second call reuses the buffers, streams and events of the first
        out.zero_()
        layer.prefill_from_host(q, k, v, out, chunk=2048)
        torch.cuda.current_stream().synchronize()
        assert torch.equal(out, want.cpu())


@pytest.mark.parametrize("T,Hq,Hkv,dh,chunk,until,sizes", [
    (1500, 8, 2, 128, 512, 640, dict(pool_size=4, bucket_size=8, bucket_cap=16, cluster_block_size=128, top_p=64, top_k=600,
                                     sink_size=4, window_size=150)),  # the picks run out first, at 64 buckets of 16 a block
    (1500, 8, 2, 128, 2048, 384, dict(pool_size=4, bucket_size=8, bucket_cap=16, cluster_block_size=128, top_p=40, top_k=640,
                                      sink_size=0, window_size=128)),  # and at 40, inside a chunk
    (1500, 8, 2, 128, 300, 384, dict(pool_size=4, bucket_size=8, bucket_cap=16, cluster_block_size=128, top_p=64, top_k=300,
                                     sink_size=4, window_size=150)),  # the key budget first: 454 keys
    (777, 5, 1, 64, 300, 1024, dict(pool_size=16, bucket_size=32, bucket_cap=64, cluster_block_size=256, top_p=64, top_k=4096,
                                    sink_size=4, window_size=256)),   # every row reads everything
    (700, 8, 2, 128, 256, 0, dict(pool_size=4, bucket_size=8, bucket_cap=16, cluster_block_size=256, top_p=64, top_k=600,
                                  sink_size=4, window_size=100)),     # a window short of a block: no row is read densely
])
def test_rows_that_read_everything_are_read_densely(oracle, T, Hq, Hkv, dh, chunk, until, sizes, monkeypatch):
    """Rows before a design leaves anything out take the dense causal read, and no others; from there on the lists: both equal
    the gather of every row's whole list, and the boundary is the whole tile of 128 rows at or before the first row whose list,
    the oracle's, leaves a key out."""
    from lsa_b200 import ops
    from lsa_b200.layer import FlatDesign

    design = FlatDesign(**sizes)
    layer, _ = _layer(Hq, Hkv, dh, 64, design, T)
    q, k, v = layer_inputs(T, Hq, Hkv, dh, 16, T + 2)
    Q, K, V = (cuda(a, torch.bfloat16) for a in (q, k, v))
    dense, read = [], ops.causal_attend

    def recorded(rows, keys, values, first, *args, **kw):
        dense.extend(range(first, first + rows.shape[0]))
        return read(rows, keys, values, first, *args, **kw)

    monkeypatch.setattr(ops, "causal_attend", recorded)
    out, index = layer.prefill(Q, K, V, chunk=chunk, return_index=True)
    assert dense == list(range(min(T, until))) and layer._whole_until(index) == until
    gathered = layer.prefill(Q, K, V, chunk=chunk, band=False, bucket_major=False)
    assert len(dense) == min(T, until)
    err = (out.float() - gathered.float()).abs()
    assert err.max() <= 2e-2 and err.mean() <= 2e-3, (err.max(), err.mean())
    index_q, index_k = layer.index_queries(Q).cpu().numpy(), index.index_keys.cpu().numpy()
    buckets = oracle.build_buckets(index_k, design.pool_size, design.bucket_size, design.bucket_cap,
                                   design.cluster_block_size)
    _, lengths = oracle.read(index_q, np.arange(T), buckets, design.top_p, design.top_k, design.sink_size, design.window_size)
    short = np.flatnonzero(lengths != np.arange(T) + 1)
    first = int(short[0]) if len(short) else T
    assert min(T, until) <= first
    if until and until < T:  # (a window that reaches past the last block's start hides the boundary for a while)
        assert first < until + design.window_size + design.cluster_block_size
    layer.check()


def test_a_selection_outlives_a_shorter_one():
    """Lists and picks handed out in the layer's own buffers are those of their shape: a call with fewer rows, and a prefill
    between, leave them as they were."""
    from lsa_b200.layer import FlatDesign

    T, Hq, Hkv = 3000, 8, 2
    design = FlatDesign(pool_size=4, bucket_size=8, bucket_cap=16, cluster_block_size=128, top_p=40, top_k=200, sink_size=4,
                        window_size=128)
    layer, _ = _layer(Hq, Hkv, 128, 64, design, 1)
    Q, K, V = (cuda(a, torch.bfloat16) for a in layer_inputs(T, Hq, Hkv, 128, 16, 1))
    index = layer.build_index(K)
    index_q, positions = layer.index_queries(Q), torch.arange(T, device="cuda")
    lists, lengths = layer.select(index_q[1000:], positions[1000:], index, reuse_buffers=True)
    picked = layer.pick(index_q[1000:], positions[1000:], index, reuse_buffers=True)[0]
    band = layer.band(Q[1000:], K, V, 1000)
    held = (lists, lengths, picked, *band)
    kept = [x.clone() for x in held]
    layer.select(index_q[500:900], positions[500:900], index, reuse_buffers=True)
    layer.pick(index_q[500:900], positions[500:900], index, reuse_buffers=True)
    layer.band(Q[500:900], K, V, 500)
    layer.prefill(Q[:1100], K[:1100], V[:1100], chunk=400)
    inside = torch.arange(lists.shape[1], device="cuda") < lengths[:, None].long()
    assert torch.equal(lists[inside], kept[0][inside])
    assert all(torch.equal(x, y) for x, y in zip(held[1:], kept[1:]))


@pytest.mark.parametrize("sizes,d_idx", [
    (dict(pool_size=16, bucket_size=32, bucket_cap=64, cluster_block_size=256, top_p=64, top_k=1024, sink_size=4,
          window_size=128), 64),
    (dict(pool_size=16, bucket_size=64, bucket_cap=128, cluster_block_size=512, top_p=16, top_k=1024, sink_size=4,
          window_size=128), 32)])
def test_prompts_that_grow_hold_no_workspace_more(sizes, d_idx, monkeypatch):
    """Layers over prompts that get longer share the bucket-major read's workspace, and none is held after a prefill; wide
    buckets without memory for one are gathered."""
    from lsa_b200 import ops
    from lsa_b200.layer import FlatDesign

    design, Hq, Hkv, chunk = FlatDesign(**sizes), 16, 4, 2048
    k, v = (torch.randn(9000, Hkv, 128, device="cuda").bfloat16() for _ in range(2))
    q = torch.randn(9000, Hq, 128, device="cuda").bfloat16()
    layers = [_layer(Hq, Hkv, 128, d_idx, design, 1)[0] for _ in range(2)]
    need = ops.bucket_attend_workspace(chunk, design.top_p, Hq, 128, 9000 // design.bucket_size, design.bucket_cap)
    torch.cuda.empty_cache()
    base, reserved = torch.cuda.memory_allocated(), torch.cuda.memory_reserved()
    out = torch.empty(9000, Hq, 128, device="cuda", dtype=torch.bfloat16)
    for T in range(5000, 9001, 500):
        for layer in layers:
            layer.prefill(q[:T], k[:T], v[:T], chunk=chunk, out=out[:T])
    own = sum(b.numel() * b.element_size() for layer in layers for held in layer._buffers.values()
              for b in (held if isinstance(held, list) else [held]))
    grown = torch.cuda.memory_allocated() - base - out.numel() * 2
    assert grown <= own + (1 << 21) * 8, (grown, own)   # (a layer's buffers, rounded up a little each)
    assert own < 18 * need // 2, (own, need)            # (eighteen prefills; no workspace is among the buffers)
    assert torch.cuda.memory_reserved() - reserved < own + out.numel() * 2 + 3 * need
    want = layers[0].prefill(q, k, v, chunk=chunk, bucket_major=False)
    empty = torch.empty

    def without(*shape, **kw):
        if kw.get("dtype") == torch.uint8:
            raise torch.OutOfMemoryError("said on the host")
        return empty(*shape, **kw)

    with monkeypatch.context() as patch:
        patch.setattr(torch, "empty", without)
        if design.bucket_cap > 64:
            assert torch.equal(layers[0].prefill(q, k, v, chunk=chunk, out=out), want)
        else:
            with pytest.raises(torch.OutOfMemoryError):
                layers[0].prefill(q, k, v, chunk=chunk, out=out)


def test_wide_buckets_write_fp32_and_take_queries_that_start_anywhere():
    """What the gather of wide buckets takes, though the bucket-major read does not: an fp32 output, and query rows at an odd
    pair of elements; the same read as the aligned bf16 call."""
    from lsa_b200.layer import FlatDesign

    T, Hq, Hkv = 3000, 8, 2
    design = FlatDesign(pool_size=16, bucket_size=64, bucket_cap=128, cluster_block_size=512, top_p=4, top_k=512, sink_size=4,
                        window_size=512)
    layer, _ = _layer(Hq, Hkv, 128, 32, design, 2)
    Q, K, V = (cuda(a, torch.bfloat16) for a in layer_inputs(T, Hq, Hkv, 128, 16, 2))
    want = layer.prefill(Q, K, V, chunk=1024)
    exact = torch.empty(T, Hq, 128, device="cuda")
    layer.prefill(Q, K, V, chunk=1024, out=exact)
    odd = torch.empty(Q.numel() + 2, device="cuda", dtype=torch.bfloat16)[2:].view(T, Hq, 128).copy_(Q)
    shifted = layer.prefill(odd, K, V, chunk=1024)
    err = (exact - want.float()).abs()
    assert err.max() <= 2e-2 and err.mean() <= 2e-3 and not torch.equal(exact, exact.bfloat16().float())
    # (rows that no tensor map can walk are mapped in fp32: another order of sums, another bucket where two scores nearly tie)
    near = (shifted.float() - want.float()).abs().amax(dim=(1, 2)) <= 2e-2
    assert near.float().mean() >= 0.98, near.float().mean()
    layer.check()
