"""One LSA global-attention layer, flat design: index build, selection and the sparse read strung together.

This is the call a serving backend makes per layer (the reference's `LayerIndex.extend` followed by
`select_and_read`, src/lsa/sglang/index/layer_index.py:824-882 and src/lsa/sglang/models/qwen3_5/backend.py:784-822),
for a single request whose KV rows sit at their positions.
"""

from __future__ import annotations

import operator
from dataclasses import dataclass

import torch

from lsa_b200 import _lib, ops, probe
from lsa_b200.budget import EarlyBudget
from lsa_b200.core import Buckets, RotaryLayout, check_sizes
from lsa_b200.shape import Shape


@dataclass(frozen=True)
class FlatDesign:
    """The sizes of a flat design (the reference's `DesignSettings`, src/lsa/sglang/settings/design.py:163-210)."""

    pool_size: int = 4
    bucket_size: int = 8
    bucket_cap: int = 16
    cluster_block_size: int = 512
    top_p: int = 1024
    top_k: int = 4096
    sink_size: int = 4
    window_size: int = 512
    early_budget: EarlyBudget | None = None
    bucket_shape: Shape | None = None  # buckets keep their spread and score as their estimated best key

    def __post_init__(self) -> None:
        check_sizes(self.pool_size, self.bucket_size, self.bucket_cap, self.cluster_block_size)
        object.__setattr__(self, "bucket_shape", Shape.read("bucket_shape", self.bucket_shape))
        if self.bucket_shape is not None and self.bucket_shape.rank > self.bucket_cap:
            raise ValueError(f"bucket_shape keeps at most bucket_cap {self.bucket_cap} directions - got rank "
                             f"{self.bucket_shape.rank}")
        if min(self.top_p, self.top_k, self.window_size) < 1 or self.sink_size < 0:
            raise ValueError("top_p, top_k and window_size must be positive and sink_size non-negative")
        if self.top_p * self.bucket_cap < self.top_k:
            raise ValueError(f"top_p {self.top_p} buckets of at most {self.bucket_cap} keys cannot fill top_k {self.top_k}")

    @property
    def block_bucket_count(self) -> int:
        return self.cluster_block_size // self.bucket_size

    @property
    def list_width(self) -> int:
        return self.top_k + self.window_size + self.sink_size

    def whole_until(self, buckets: int) -> int:
        """The first position whose read leaves anything out, over an index of `buckets` buckets. A row before it picks
        every bucket it sees, no cut bites, and the window covers what is in no closed block yet: its list is all the keys
        up to its own, so a dense causal read is the same read (and scores, picks and lists nothing). 0 where a design has
        no such rows; else whole tiles of 128 query rows."""
        if self.window_size < self.cluster_block_size or self.early_budget is not None:
            return 0
        by_buckets = (min(self.top_p, buckets) // self.block_bucket_count + 1) * self.cluster_block_size
        return min(by_buckets, self.list_width) // 128 * 128


class FlatIndex:
    """A request's index: its index keys and the buckets of its closed cluster blocks (and, where the tensor-core
    scan can use it, its operand: the centroids less a common centre in bf16, and the greatest length of one)."""

    def __init__(self, index_keys: torch.Tensor, buckets: Buckets, centroids_bf16: torch.Tensor | None = None,
                 lengths: torch.Tensor | None = None, radius: torch.Tensor | None = None,
                 shapes: ops.ShapeTable | None = None):
        self.index_keys = index_keys
        self.buckets = buckets
        self.centroids_bf16 = centroids_bf16
        self.lengths, self.radius = lengths, radius
        self.shapes = shapes  # the buckets' shapes, row for row, under a design with `bucket_shape`


class FlatLayer:
    """Prefill and decode of one layer. `query_map` / `key_map` are [Hkv * (dh - rotary), index_dim]."""

    def __init__(self, design: FlatDesign, query_map: torch.Tensor, key_map: torch.Tensor, heads: int, kv_heads: int,
                 head_dim: int, rotary: RotaryLayout = RotaryLayout(), scale: float | None = None,
                 tensor_cores: bool = True):
        if heads % kv_heads:
            raise ValueError(f"query heads must group evenly - {heads} does not divide by {kv_heads}")
        free = head_dim - rotary.dim
        if query_map.shape != key_map.shape or query_map.shape[0] != kv_heads * free:
            raise ValueError(f"the maps must both be [{kv_heads * free}, index_dim] - got {tuple(query_map.shape)} "
                             f"and {tuple(key_map.shape)}")
        self.design = design
        self.index_dim = key_map.shape[1]
        self.query_map, self.key_map = query_map.contiguous(), key_map.contiguous()
        self.heads, self.kv_heads, self.head_dim = heads, kv_heads, head_dim
        self.dh_off = rotary.dim if rotary.end == "prefix" else 0
        self.dh_used = free
        self.scale = head_dim ** -0.5 if scale is None else scale
        self._buffers: dict = {}
        # What the kernels report from the device, read by `check()`: bounded waits of the map kernels that gave up,
        # buckets over their cap in the table, bad picks in the expansion, bounded waits of the attention kernels.
        self._status_slots(query_map.device)
        self._reached: list = []  # per index build: whether each cluster block merged down to its bucket count
        # The bucket-major attend pass has two forms: (pair, head) rows as the M = 128 side of tcgen05 products with S
        # and O in tensor memory (the default), or warp-level MMA tiles of 16 rows.
        self.bucket_tensor_memory = True
        self._band_stream = self._band_done = None  # the side stream the band runs on beside the bucket-major read
        self._copy_in = self._copy_out = self._index_stream = None  # the side streams of `prefill_from_host`
        self._copy_events: list = []
        # bf16 maps run on the tensor cores (the head sum folded into the product); fp32 maps keep the exact form
        self.tensor_cores = tensor_cores and query_map.dtype == torch.bfloat16 and key_map.dtype == torch.bfloat16 \
            and query_map.shape[1] in (32, 64, 128)
        if self.tensor_cores:
            self.query_map_t = ops.expand_map(self.query_map, heads, heads // kv_heads, head_dim, self.dh_off,
                                              self.dh_used)
            self.key_map_t = ops.expand_map(self.key_map, kv_heads, 1, head_dim, self.dh_off, self.dh_used)

    def _status_slots(self, device) -> None:
        """The layer's deferred-status words: index map, bucket table, expansion, attention, bucket scan."""
        self.status = torch.zeros(5, device=device, dtype=torch.int32)
        self._map_status, self._table_status = self.status[0:1], self.status[1:2]
        self._expand_status, self._attend_status = self.status[2:3], self.status[3:4]
        self._scan_status = self.status[4:5]

    def check(self) -> None:
        """The deferred checks of everything launched since the last call: ONE host synchronisation, so a hot path
        calls it once a prefill (or once a benchmark) rather than after every kernel. Raises `ValueError` when a
        cluster block stopped short of its bucket count or a bucket overflowed its cap (what `core.build_buckets`
        raises at once, src/lsa/core/reference.py:131, ward.py:118-122) and `RuntimeError` when a bounded on-chip
        wait gave up, in which case the outputs since the last check are void."""
        counts = self.status.tolist()
        short = sum(int((~r.bool()).sum()) for r in self._reached)
        self.status.zero_()
        self._reached.clear()
        if short or counts[1]:
            raise ValueError(f"{short} cluster blocks stopped short of {self.design.block_bucket_count} buckets under "
                             f"the cap {self.design.bucket_cap}; {counts[1]} buckets overflowed it")
        if counts[2]:
            raise ValueError(f"{counts[2]} picked bucket ids lay outside the member table")
        if counts[0] or counts[3] or counts[4]:
            raise RuntimeError(f"bounded on-chip waits gave up ({counts[0]} in the index map, {counts[3]} in the "
                               f"attention kernels, {counts[4]} in the bucket scan): the outputs since the last "
                               "check are void")

    # ---- buffers

    def _buffer(self, name: str, shape: tuple, dtype: torch.dtype, device) -> torch.Tensor:
        """A tensor that lives as long as the layer, one a shape: what a call hands out stays until the next call of that
        shape, and a step allocates nothing once every shape has been seen."""
        key = (name, tuple(shape), dtype, str(device))
        held = self._buffers.get(key)
        if held is None:
            held = self._buffers[key] = torch.empty(shape, device=device, dtype=dtype)
        return held

    def _room(self, name: str, shape: tuple, dtype: torch.dtype, device) -> torch.Tensor:
        """The same for what no call hands out: the leading rows of a buffer of that name, so that a ragged chunk allocates
        nothing beside a whole one. A buffer that is outgrown stays (a captured graph may hold its address) and the next has
        half as many rows again, where there is memory for that: all of a name's are less than five times the largest asked
        for."""
        held = self._buffers.setdefault((name, "rows", tuple(shape[1:]), dtype, str(device)), [])
        for buffer in held:
            if buffer.shape[0] >= shape[0]:
                return buffer[:shape[0]]
        rows = max(shape[0], held[-1].shape[0] * 3 // 2) if held else shape[0]
        try:
            held.append(torch.empty(rows, *shape[1:], device=device, dtype=dtype))
        except torch.OutOfMemoryError:
            if rows == shape[0]:
                raise
            held.append(torch.empty(shape, device=device, dtype=dtype))
        return held[-1][:shape[0]]

    def _takes_tensor_cores(self, x: torch.Tensor) -> bool:
        """Heads packed densely in bf16 with a 16-byte aligned row pitch: the layout a TMA descriptor can walk."""
        # (a handful of rows - a decode step - goes to the kernel that splits one row's contraction over a CTA)
        return (self.tensor_cores and x.shape[0] > 32 and x.dtype == torch.bfloat16 and x.stride(2) == 1
                and x.stride(1) == x.shape[2]
                and x.stride(0) % 8 == 0 and x.data_ptr() % 16 == 0)

    # ---- the stages

    few_rows = 128  # up to this many queries are mapped a CTA a row (5.4 us for 128 of 5,120 dims; one tile of a GEMM 26.8)

    def index_queries(self, q: torch.Tensor, out: torch.Tensor | None = None) -> torch.Tensor:
        """q [T, Hq, dh] bf16 -> unit index queries [T, index_dim] fp32."""
        if q.shape[0] > self.few_rows and self._takes_tensor_cores(q):
            return ops.index_map_tc(q, self.query_map_t, out=out, status=self._map_status)
        return ops.index_map(q, self.query_map, group=self.heads // self.kv_heads, dh_off=self.dh_off,
                             dh_used=self.dh_used, out=out)

    def index_queries_rows(self, q: torch.Tensor) -> torch.Tensor:
        """The same map for the few rows of a decode step, q [R <= 8, Hq, dh] bf16: `index_queries`, whose kernel for few rows sums a
        KV head's group before it multiplies (one row of 40 heads over 8: 5.0 us and one launch, where a map of all 40 heads'
        dims, a fifth of them read as often, took 5.7 and 1.9 for the unit length)."""
        return self.index_queries(q)

    def index_keys(self, k: torch.Tensor, out: torch.Tensor | None = None) -> torch.Tensor:
        """k [T, Hkv, dh] bf16 -> unit index keys [T, index_dim] fp32."""
        if self._takes_tensor_cores(k):
            return ops.index_map_tc(k, self.key_map_t, out=out, status=self._map_status)
        return ops.index_map(k, self.key_map, group=1, dh_off=self.dh_off, dh_used=self.dh_used, out=out)

    def build_index(self, k: torch.Tensor, reuse_buffers: bool = False) -> FlatIndex:
        """Index keys, then pools, Ward and the bucket table of every closed cluster block.

        With `reuse_buffers` the index lives in the layer's own buffers and is overwritten by the next build.
        """
        bufs = self._index_buffers(k.shape[0], k.device, reuse_buffers)
        self._build_blocks(k, 0, bufs)
        return self._index_of(bufs)

    def _index_buffers(self, T: int, dev, reuse_buffers: bool) -> dict:
        """The tensors an index over T keys lives in (the layer's own buffers, or fresh ones)."""
        d, d_idx = self.design, self.index_dim
        blocks = T // d.cluster_block_size
        P, rows = d.cluster_block_size // d.pool_size, blocks * d.block_bucket_count
        make = (lambda name, shape, dtype: self._buffer(name, shape, dtype, dev)) if reuse_buffers else \
            (lambda name, shape, dtype: torch.empty(shape, device=dev, dtype=dtype))
        bufs = {"keys": make("index keys", (T, d_idx), torch.float32),
                "pools": make("pools", (blocks, P, d_idx), torch.float32),
                "labels": make("labels", (blocks, P), torch.int64), "reached": make("reached", (blocks,), torch.uint8),
                "status": self._table_status,
                "members": make("members", (rows, d.bucket_cap), torch.int32), "sizes": make("sizes", (rows,), torch.int32),
                "key sums": make("key sums", (rows, d_idx), torch.float32),
                "centroids": make("centroids", (rows, d_idx), torch.float32)}
        if d_idx == 64:  # (the operand of the tensor-core scan: centroids less the first blocks' mean, in bf16)
            bufs["centroids bf16"] = make("centroids bf16", (rows, d_idx), torch.bfloat16)
            bufs["centre"], bufs["radius"] = make("centre", (d_idx,), torch.float32), make("radius", (1,), torch.float32)
            bufs["lengths"] = make("operand lengths", (rows,), torch.float32)
            bufs["radius"].zero_()
            bufs["centred"] = [False]
        if d.bucket_shape is not None:
            if d_idx not in (32, 64):
                raise ValueError(f"bucket shapes are built over index keys of 32 or 64 dims - got {d_idx}")
            rank = d.bucket_shape.rank
            bufs["shapes"] = ops.ShapeTable(make("shape basis", (rows, rank, d_idx // 8), torch.uint8),
                                            make("shape variances", (rows, rank), torch.float32),
                                            make("shape floor", (rows,), torch.float32), d.bucket_shape.deviations)
        return bufs

    def _index_of(self, bufs: dict) -> FlatIndex:
        d = self.design
        return FlatIndex(bufs["keys"], Buckets(bufs["centroids"], bufs["members"], bufs["sizes"], d.block_bucket_count,
                                               d.cluster_block_size), bufs.get("centroids bf16"), bufs.get("lengths"),
                         bufs.get("radius"), bufs.get("shapes"))

    def _build_blocks(self, k: torch.Tensor, first: int, bufs: dict) -> None:
        """Index keys of k [n, ...] = the keys at positions first.., and the pools, Ward labels and bucket table of
        the cluster blocks they close (first is a multiple of the block size): blocks are independent, so an index
        can be built as its keys arrive."""
        d = self.design
        n = k.shape[0]
        with probe.region("index map"):
            self.index_keys(k, out=bufs["keys"][first:first + n])
        self._cluster_blocks(first // d.cluster_block_size, n // d.cluster_block_size, bufs)

    def _cluster_blocks(self, b0: int, nb: int, bufs: dict) -> None:
        """Pools, Ward labels and the bucket table of cluster blocks b0 .. b0 + nb - 1, whose index keys are in place."""
        d = self.design
        if nb <= 0:
            return
        first = b0 * d.cluster_block_size
        r0, r1 = b0 * d.block_bucket_count, (b0 + nb) * d.block_bucket_count
        keys = bufs["keys"][first:first + nb * d.cluster_block_size]
        with probe.region("pool"):
            pools = ops.pool_keys(keys.view(nb, d.cluster_block_size, -1), d.pool_size, out=bufs["pools"][b0:b0 + nb])
        with probe.region("ward"):
            labels, _ = ops.ward_rounds(pools, float(d.pool_size), d.block_bucket_count, d.bucket_cap,
                                        labels=bufs["labels"][b0:b0 + nb], reached=bufs["reached"][b0:b0 + nb])
            if len(self._reached) < 64:  # (views of the index buffers; `check()` reads and drops them)
                self._reached.append(bufs["reached"][b0:b0 + nb])
        with probe.region("bucket table"):
            outs = (bufs["members"][r0:r1], bufs["sizes"][r0:r1], bufs["key sums"][r0:r1], bufs["centroids"][r0:r1],
                    None, bufs["status"])
            ops.bucket_table(keys, labels, d.pool_size, d.block_bucket_count, d.bucket_cap, first_position=first,
                             outs=outs)
            if "centroids bf16" in bufs:
                # Any centre leaves the ranking as it is; the mean of the first blocks' centroids is where the cone
                # of this layer's index vectors points, and the closer to it the rows lie, the sharper the scan.
                if not bufs["centred"][0]:
                    bufs["centre"].copy_(bufs["centroids"][r0:r1].mean(0))
                    bufs["centred"][0] = True
                ops.scan_centre(bufs["centroids"][r0:r1], bufs["centre"], bufs["centroids bf16"][r0:r1],
                                bufs["lengths"][r0:r1], bufs["radius"])
        if "shapes" in bufs:  # (members are positions: the keys of these blocks start at `first`)
            with probe.region("bucket shapes"):
                ops.shape_build(keys, bufs["centroids"][r0:r1], bufs["members"][r0:r1], d.bucket_shape.rank,
                                key_base=first, out=bufs["shapes"].rows(slice(r0, r1)))

    scan_rows = 1024  # from this many rows on, a pick over more than 4,096 buckets in sight runs its scan on the tensor cores

    def pick(self, index_queries: torch.Tensor, positions: torch.Tensor, index: FlatIndex,
             reuse_buffers: bool = False, last_position: int | None = None):
        """The top-p buckets of every row, best first: (picked [R, top_p] int32, positions int64, and the rows' own
        budgets under an early budget, else None). `last_position` is the host's bound on `positions`, if it has
        one: no position is past it, and no bucket that it does not see is searched (nor a sample of the tensor-core scan taken
        there); the result is the same under any such bound."""
        return self._pick(index_queries, positions, index, self._buffer if reuse_buffers else None, last_position)

    def _pick(self, index_queries: torch.Tensor, positions: torch.Tensor, index: FlatIndex, held, last_position: int | None):
        """`pick` into what `held` (`_buffer` or `_room`) gives, or into fresh tensors."""
        d, b, dev = self.design, index.buckets, index_queries.device
        R = index_queries.shape[0]
        positions = positions.to(torch.int64)
        visible = ops.visible_buckets(positions, d.cluster_block_size, d.block_bucket_count, b.bucket_centroids.shape[0])
        row_p = row_k = None
        if d.early_budget is not None:
            early = positions < d.early_budget.position
            row_p = torch.where(early, d.early_budget.top_p, d.top_p).to(torch.int32)
            row_k = torch.where(early, d.early_budget.top_k, d.top_k).to(torch.int32)
        keys = picked = None
        if held is not None:
            keys = held("keys", (R, d.top_p), torch.int64, dev)
            picked = held("picked", (R, d.top_p), torch.int32, dev)
        with probe.region("select"):
            bound = 0 if last_position is None else last_position // d.cluster_block_size * d.block_bucket_count
            bound = min(bound or b.bucket_centroids.shape[0], b.bucket_centroids.shape[0])
            # (the scan's threshold rests on 512 samples of a row's scores: it needs the kept ones to be a fair share of the
            # buckets in sight - else the exact search, at once. That one places a row's best out of 4,096 scores in 0.22 ms a chunk
            # of 8,192 rows, and of fewer in less, where the scan's launches take 0.24 whatever is in sight)
            if index.shapes is not None:  # a bucket scores as its estimated best key: the exact scan, shaped
                _, picked = ops.shaped_select(index_queries, b.bucket_centroids, index.shapes, visible, d.top_p, row_p,
                                              keys=keys, picked=picked)
            elif index.centroids_bf16 is not None and R >= self.scan_rows and d.top_p <= 512 and bound > ops.BINNED_BUCKETS \
                    and 3 * d.top_p * 512 >= 8 * bound:
                need = ops.query("lsa_scan_select_workspace_bytes", R, d.top_p, b.bucket_centroids.shape[0])
                work = self._room("scan", (need,), torch.uint8, dev)
                _, picked = ops.scan_select(index_queries, b.bucket_centroids, index.centroids_bf16, visible, d.top_p,
                                            row_p, max_visible=bound, keys=keys, picked=picked,
                                            status=self._scan_status, workspace=work, lengths=index.lengths,
                                            radius=index.radius)
            elif R <= 8 and row_p is None and d.top_p <= 128 and keys is None and b.bucket_centroids.shape[1] in (32, 64):
                _, picked = ops.flat_select_decode(index_queries, b.bucket_centroids, None, visible, d.top_p,
                                                   splits=self._decode_splits(R, b.bucket_centroids.shape[0]))
            else:  # (of the buckets that the last row sees: no row sees one past them)
                _, picked = ops.flat_select(index_queries, b.bucket_centroids[:bound], visible, d.top_p, row_p, keys=keys,
                                            picked=picked)
        return picked, positions, row_p, row_k

    def select(self, index_queries: torch.Tensor, positions: torch.Tensor, index: FlatIndex,
               reuse_buffers: bool = False, local: bool = True, last_position: int | None = None):
        """Read lists [R, top_k + window + sink] int32 and their lengths for queries at `positions`; with
        `local=False` the lists hold the expansion alone (a band kernel reads the window and the sinks)."""
        return self._select(index_queries, positions, index, self._buffer if reuse_buffers else None, local, last_position)

    def _select(self, index_queries: torch.Tensor, positions: torch.Tensor, index: FlatIndex, held, local: bool,
                last_position: int | None):
        """`select` into what `held` gives, or into fresh tensors."""
        d, b, dev = self.design, index.buckets, index_queries.device
        R = index_queries.shape[0]
        picked, positions, row_p, row_k = self._pick(index_queries, positions, index, held, last_position)
        if held is not None:
            lists, lengths = held("lists", (R, d.list_width), torch.int32, dev), held("lengths", (R,), torch.int32, dev)
        else:
            lists = torch.empty(R, d.list_width, device=dev, dtype=torch.int32)
            lengths = torch.empty(R, device=dev, dtype=torch.int32)
        with probe.region("expand"):
            # (the layer's own buffers are read by their lengths: nothing is padded there)
            lists, lengths, _ = ops.expand(picked, positions, b.bucket_members, d.top_k, d.sink_size, d.window_size,
                                           row_p, row_k, outs=(lists, lengths, self._expand_status), local=local,
                                           pad=held is None)
        return lists, lengths

    def attend(self, q: torch.Tensor, k: torch.Tensor, v: torch.Tensor, lists: torch.Tensor, lengths: torch.Tensor,
               splits: int = 1, out: torch.Tensor | None = None, lse: torch.Tensor | None = None,
               init: tuple | None = None):
        with probe.region("attend"):
            return ops.sparse_attend(q, k, v, lists, lengths, self.scale, splits=splits, out=out, lse=lse, init=init)

    def band(self, q: torch.Tensor, k: torch.Tensor, v: torch.Tensor, first_position: int):
        """The window and sinks of consecutive rows as one dense banded read: a partial (out fp32, lse)."""
        return self._band(q, k, v, first_position, *self._partial(self._buffer, "band", q.shape[0], q.device))

    def _partial(self, held, name: str, rows: int, device) -> tuple:
        """A partial read's tensors: out fp32 and lse."""
        return (held(f"{name} out", (rows, self.heads, self.head_dim), torch.float32, device),
                held(f"{name} lse", (rows, self.heads), torch.float32, device))

    def _band(self, q: torch.Tensor, k: torch.Tensor, v: torch.Tensor, first_position: int, out: torch.Tensor,
              lse: torch.Tensor):
        with probe.region("band"):
            return ops.band_attend(q, k, v, first_position, self.design.window_size, self.design.sink_size, self.scale,
                                   out=out, lse=lse, status=self._attend_status)

    # ---- the layer

    def prefill(self, q: torch.Tensor, k: torch.Tensor, v: torch.Tensor, chunk: int = 8192,
                return_index: bool = False, out: torch.Tensor | None = None, band: bool = True,
                bucket_major: bool = True):
        """Causal prefill from position 0: q [T,Hq,dh], k/v [T,Hkv,dh] bf16 -> out [T,Hq,dh] bf16.

        Every intermediate lives in buffers the layer keeps, but for what is the allocator's again after each chunk: the bucket-major
        read's workspace, the masks and the exact search's scores (48 MiB at most). After the first call a step allocates nothing
        beside those and its output (pass `out` to avoid that too). With `return_index` the index is built in fresh tensors instead.
        `band` reads the window and the sinks as dense tiles; `bucket_major` reads the selected keys bucket by bucket
        where the shapes allow and it is the faster read (both off: every row gathers its whole list).

        `chunk` is how many rows are worked on at a time, and with that how large the buffers get. Rows that are read through
        masks (`_listed_until`) are taken two waves of the GPU at a time where that is more, their tensors are what the masked
        read takes and there is memory for it; else, as all others, `chunk` at a time. Which keys a row lists depends on its
        position and not on the chunk it is in, but for buckets whose scores nearly tie: a last piece of up to 128 rows is mapped in
        fp32, larger ones on the tensor cores (and a piece of fewer than 128 rows is not read through masks).
        """
        T = q.shape[0]
        index = self.build_index(k, reuse_buffers=not return_index)
        out = torch.empty_like(q) if out is None else out
        whole = min(T, self._whole_until(index)) if band else 0  # (rows that read everything make chunks of their own)

        def read(first: int, end: int) -> None:
            for start in range(first, end, chunk):
                stop = min(end, start + chunk)
                self.prefill_rows(q[start:stop], start, k, v, index, out[start:stop], band, bucket_major)

        read(0, whole)
        first = whole
        if band and bucket_major and ops.dense_attend_supported(q, k, v, out) and whole < min(T, self._listed_until()):
            # (a CTA of the masked read has 256 rows of a head: chunks of fewer than two waves leave part of the GPU idle, 24,576
            # tokens of 8 heads in chunks of 2,048 rows 7.1 ms and 4.8 this way)
            sms = torch.cuda.get_device_properties(q.device).multi_processor_count
            step = max(chunk, -(-2 * sms * 256 // self.heads // 128) * 128)
            listed = min(T, self._listed_until())
            for first in range(whole, listed, step):
                stop = min(listed, first + step)
                if stop - first <= chunk or not self._reads_wide(q[first:stop], first, k, v, index, out[first:stop]):
                    read(first, stop)
            first = listed
        read(first, T)
        return (out, index) if return_index else out

    def prefill_from_host(self, q_host: torch.Tensor, k_host: torch.Tensor, v_host: torch.Tensor,
                          out_host: torch.Tensor, chunk: int = 8192) -> torch.Tensor:
        """`prefill` for inputs and an output that live in PINNED host memory, the copies overlapped with the work.
        A causal chunk needs the keys and values up to its own end and the buckets of the cluster blocks before its
        rows, and blocks are clustered independently: so K, V and Q cross chunk by chunk on a copy stream, each
        chunk's blocks are indexed when its keys have arrived (on a stream of its own: a handful of small launches
        that would otherwise stand between two chunks' reads), and every chunk's output leaves on a second copy
        stream as soon as its merge is done. (`chunk` must hold whole cluster blocks.) On return the current stream
        has waited for the last output copy; synchronise it before reading `out_host`."""
        dev = self.query_map.device
        T = q_host.shape[0]
        if chunk % self.design.cluster_block_size or chunk % 128:
            raise ValueError("a chunk must hold whole cluster blocks (and whole tiles of 128 keys)")
        main = torch.cuda.current_stream(dev)
        if self._copy_in is None:
            self._copy_in, self._copy_out, self._index_stream = (torch.cuda.Stream(dev) for _ in range(3))
        chunks = [(start, min(T, start + chunk)) for start in range(0, T, chunk)]
        while len(self._copy_events) < 3 * len(chunks):
            self._copy_events.append(torch.cuda.Event())
        arrived, done, built = self._copy_events[0::3], self._copy_events[1::3], self._copy_events[2::3]
        q = self._room("q from host", tuple(q_host.shape), q_host.dtype, dev)
        k = self._room("k from host", tuple(k_host.shape), k_host.dtype, dev)
        v = self._room("v from host", tuple(v_host.shape), v_host.dtype, dev)
        out = self._room("out to host", tuple(q_host.shape), torch.bfloat16, dev)
        self._copy_in.wait_stream(main)   # the last call's reads of these buffers are over
        self._copy_out.wait_stream(main)
        with torch.cuda.stream(self._copy_in):
            for c, (start, stop) in enumerate(chunks):
                k[start:stop].copy_(k_host[start:stop], non_blocking=True)
                v[start:stop].copy_(v_host[start:stop], non_blocking=True)
                q[start:stop].copy_(q_host[start:stop], non_blocking=True)
                arrived[c].record(self._copy_in)
        bufs = self._index_buffers(T, dev, reuse_buffers=True)
        index = self._index_of(bufs)
        self._index_stream.wait_stream(main)
        with torch.cuda.stream(self._index_stream):
            for c, (start, stop) in enumerate(chunks):
                self._index_stream.wait_event(arrived[c])
                self._build_blocks(k[start:stop], start, bufs)
                built[c].record(self._index_stream)
        for c, (start, stop) in enumerate(chunks):
            main.wait_event(built[c])  # (the chunk's keys, values and queries have arrived, and its blocks are indexed)
            # (the cache as far as it has arrived: no kernel is handed rows that are still on their way)
            self.prefill_rows(q[start:stop], start, k[:stop], v[:stop], index, out[start:stop])
            done[c].record(main)
            with torch.cuda.stream(self._copy_out):
                self._copy_out.wait_event(done[c])
                out_host[start:stop].copy_(out[start:stop], non_blocking=True)
        main.wait_stream(self._copy_out)
        return out_host

    def _whole_until(self, index: FlatIndex) -> int:
        return self.design.whole_until(index.buckets.bucket_centroids.shape[0])

    @property
    def _reads_by_bucket(self) -> bool:
        """Whether reading the selected keys bucket by bucket is the faster read. It costs a partial output a (row, pick,
        query head), whatever the bucket holds; the gather costs the bytes of a pick's keys once a KV head. Measured on a
        B200, bucket-major against gather, whole prefills: buckets of 8 keys under groups of 4, 8 and 5 heads 16.9 / 12.0,
        26.8 / 12.3 and 62.5 / 35.9 ms (24,576 tokens); buckets of 32 keys under groups of 4, 5 and 8 heads 18.1 / 32.3,
        62.3 / 144.8 and 27.4 / 34.7 ms (131,072 tokens); of 64 keys under groups of 4 2.2 / 3.3 ms (24,576 tokens): the two
        meet near three keys a query head of the group."""
        return self.design.bucket_size >= 3 * (self.heads // self.kv_heads)

    def _bucket_takes(self, rows: torch.Tensor, out: torch.Tensor) -> bool:
        """Whether wide buckets may be read bucket by bucket here: the gather, which serves them too, also writes fp32 and
        takes query rows that are not 16-byte aligned."""
        return self.design.bucket_cap <= 64 or (out.dtype == torch.bfloat16 and rows.stride(0) % 8 == 0
                                                and rows.stride(1) % 8 == 0 and rows.data_ptr() % 16 == 0)

    def _bucket_workspace(self, rows: int, index: FlatIndex, device) -> torch.Tensor | None:
        """The bucket-major read's workspace, a partial output a (row, pick, head): gigabytes that the layer does not keep. It
        goes back to the allocator with the chunk and serves the next, and the other layers of a model. Sizes are cut to 32
        steps an octave, so that an index with a few buckets more asks for the same bytes. Buckets of more than 64 members,
        which the gather served alone before there was a pass for them, go to the gather again where the workspace is over
        8 GiB or there is no memory for it. (24,576 tokens of 40 heads, 48 picks of 64 keys: 14.4 ms with 8.1 GB, in shorter
        chunks 14.9 with 4.0 and 18.0 with 1.0; the gather 25.6 to 28.3. The line keeps a chunk from a tenth of the GPU.)"""
        members = index.buckets.bucket_members
        need = ops.bucket_attend_workspace(rows, self.design.top_p, self.heads, self.head_dim, *members.shape)
        wide = members.shape[1] > 64
        if wide and need > 8 << 30:
            return None
        step = max(1 << 21, 1 << max(0, need.bit_length() - 6))
        try:
            return torch.empty(-(-need // step) * step, device=device, dtype=torch.uint8)
        except torch.OutOfMemoryError:
            if wide:
                return None
            raise

    def _listed_until(self) -> int:
        """The position up to which a row's list is read as a mask over every key before it (`ops.listed_attend`): where that
        costs what the other reads do. Measured on a B200, in ps a row and query head: a key of the masked read 0.68, so a
        row's cost grows with its position; a pick read bucket by bucket 140 (partials in bf16; 420 where buckets hold more
        than 64 members and they are fp32) and a key of the band beside it 1.2; a key of a gathered list 48 a KV head, and 10
        for its place in the list. Whole prefills, the other reads against this one up to the line: 20,011 tokens of 32 heads
        over 8, 64 picks of 32 keys 6.2 / 4.8 ms; 16,384 of 8 over 2, 16 picks of 64 keys 1.33 / 1.05; 24,576 of 8 over 2,
        4,096 keys of 1,024 picks 12.1 / 4.8."""
        d, group = self.design, self.heads // self.kv_heads
        cost = 1.2 * (d.window_size + d.sink_size)
        if self._reads_by_bucket:
            cost += d.top_p * (140 if d.bucket_cap <= 64 else 420)
        else:
            cost += d.top_k * (48 + 10 / self.kv_heads) / group
        return min(int(cost / 0.68), self.most_listed) // 128 * 128

    most_listed = 1600 * 128  # positions whose bits `ops.list_bits` holds in a CTA's shared memory, eight rows of them

    def _list_masks(self, rows: torch.Tensor, start: int, k: torch.Tensor):
        """Memory for the masks of a chunk that is read through them ([key tiles, rows, 4] int32, the allocator's again after the
        chunk); None for one that is not: rows past `_listed_until`, too few of them for its tiles, or no memory. (The caller has
        asked whether the dense read takes the tensors.)"""
        n = rows.shape[0]
        stop = start + n
        if n < 128 or start >= self._listed_until() or stop > self.most_listed or k.shape[0] < stop:
            return None
        try:
            return torch.empty(-(-stop // 128) * n * 16, device=rows.device, dtype=torch.uint8).view(torch.int32).view(-1, n, 4)
        except torch.OutOfMemoryError:
            return None

    def _read_listed(self, rows: torch.Tensor, start: int, k: torch.Tensor, v: torch.Tensor, index: FlatIndex,
                     out: torch.Tensor, mask: torch.Tensor) -> torch.Tensor:
        """The masked read of rows that `_list_masks` gave `mask` for."""
        d = self.design
        index_queries, positions = self._query_rows(rows, start)
        picked, positions, row_p, row_k = self._pick(index_queries, positions, index, self._room, start + rows.shape[0] - 1)
        with probe.region("expand"):
            ops.list_bits(picked, positions, index.buckets.bucket_members, d.top_k, d.sink_size, d.window_size, k.shape[0],
                          mask.shape[0], row_p, row_k, self._expand_status, out=mask)
        with probe.region("attend"):
            return ops.listed_attend(rows, k, v, start, mask, self.scale, out, self._attend_status)

    def _reads_wide(self, rows: torch.Tensor, start: int, k: torch.Tensor, v: torch.Tensor, index: FlatIndex,
                    out: torch.Tensor) -> bool:
        """A chunk of more rows than the caller asked for, read through masks; False where there is no memory for it."""
        mask = self._list_masks(rows, start, k)
        if mask is None:
            return False
        try:
            self._read_listed(rows, start, k, v, index, out, mask)
        except torch.OutOfMemoryError:
            return False
        return True

    def _query_rows(self, rows: torch.Tensor, start: int) -> tuple:
        """Index queries and positions of consecutive rows at positions start.."""
        n, dev = rows.shape[0], rows.device
        positions = torch.arange(start, start + n, device=dev)
        with probe.region("index map"):
            return self.index_queries(rows, out=self._room("index queries", (n, self.index_dim), torch.float32, dev)), positions

    def prefill_rows(self, rows: torch.Tensor, start: int, k: torch.Tensor, v: torch.Tensor, index: FlatIndex,
                     out: torch.Tensor, band: bool = True, bucket_major: bool = True) -> torch.Tensor:
        """The read of consecutive query rows [n, Hq, dh] at positions start.. over a cache whose index is built,
        into `out` [n, Hq, dh] bf16 - one chunk of a prefill, or one rank's rows of a chunk."""
        n, dev = rows.shape[0], rows.device
        stop = start + n
        if band and self.design.sink_size <= 64 and k.shape[0] >= stop and start < self._whole_until(index):
            # (a tensor-core row costs 0.6 ps a key and head here: 0.07 us for the 3,000 keys of a row of 40 heads, against
            # 0.5 us for its window and 64 picked buckets. The probabilities go in as two bf16 terms: the lists' read, which this
            # stands for, is closer to the sums in 64 bits than one rounded term a key.)
            whole = min(n, self._whole_until(index) - start)
            with probe.region("band"):
                partial, into = None, out[:whole]
                if whole < 128 or not ops.dense_attend_supported(rows[:whole], k, v, into):
                    partial = self._partial(self._room, "dense", whole, dev)
                    if not into.is_contiguous() or into.dtype not in (torch.bfloat16, torch.float32):
                        into = partial[0]
                ops.causal_attend(rows[:whole], k, v, start, self.scale, out=into, partial=partial,
                                  status=self._attend_status)
                if partial is not None and into is partial[0]:
                    out[:whole].copy_(into)
            if whole == n:
                return out
            self.prefill_rows(rows[whole:], start + whole, k, v, index, out[whole:], band, bucket_major)
            return out
        masked = band and bucket_major and ops.dense_attend_supported(rows, k, v, out)
        listed = self._listed_until() - start
        if masked and 0 < listed < n:  # (the rows past the line have the other reads)
            self.prefill_rows(rows[:listed], start, k, v, index, out[:listed], band, bucket_major)
            self.prefill_rows(rows[listed:], start + listed, k, v, index, out[listed:], band, bucket_major)
            return out
        mask = self._list_masks(rows, start, k) if masked else None
        if mask is not None:
            return self._read_listed(rows, start, k, v, index, out, mask)
        index_queries, positions = self._query_rows(rows, start)
        # The window and the sinks are the same keys for neighbouring rows: one dense band serves them, and the
        # read of the selected keys starts from its partial result.
        banded = band and self.design.sink_size <= 64 and k.shape[0] >= stop
        lse = self._room("lse", (n, self.heads), torch.float32, dev)
        partial = self._partial(self._room, "band", n, dev) if banded else None
        # (without the band the window and the sinks are in the lists, which only the gather path reads)
        workspace = None
        if banded and bucket_major and self._reads_by_bucket and self._bucket_takes(rows, out) and \
                ops.bucket_attend_supported(rows, k, self.design.bucket_cap, self.design.top_p,
                                            not self.bucket_tensor_memory):
            workspace = self._bucket_workspace(n, index, dev)
        if workspace is not None:
            # The band and the read of the selected keys meet only in the merge, and one waits on the tensor pipe
            # while the other is bound by instruction issue: the band runs on a stream of its own beside them.
            main = torch.cuda.current_stream(dev)
            if self._band_stream is None:
                self._band_stream, self._band_done = torch.cuda.Stream(dev), torch.cuda.Event()
            self._band_stream.wait_stream(main)  # the inputs are ready; the last chunk's merge has read the buffers
            with torch.cuda.stream(self._band_stream):
                init = self._band(rows, k, v, start, *partial)
                self._band_done.record(self._band_stream)
            # The rows of a chunk pick the same buckets over and over: read each bucket's keys once per 128
            # (row, pick) pairs instead of once per pair.
            picked, positions, row_p, row_k = self._pick(index_queries, positions, index, self._room, stop - 1)
            with probe.region("attend"):
                ops.bucket_attend(rows, k, v, picked, positions, index.buckets.bucket_members, self.design.top_k,
                                  self.design.sink_size, self.design.window_size, self.scale, init=init,
                                  row_top_p=row_p, row_top_k=row_k, out=out, lse=lse,
                                  warp_mma=not self.bucket_tensor_memory, init_ready=self._band_done,
                                  status=self._attend_status,
                                  workspace=workspace)
            return out
        init = self._band(rows, k, v, start, *partial) if banded else None
        lists, lengths = self._select(index_queries, positions, index, self._room, not banded, stop - 1)
        self.attend(rows, k, v, lists, lengths, out=out, lse=lse, init=init)
        return out

    @staticmethod
    def _decode_splits(rows: int, buckets: int) -> int:
        """CTAs that a decode row's buckets are split over: one ranks 256 at a time; up to 4,096 go to the eight CTAs of a cluster,
        more to several clusters and a merge (one row over 512 buckets: 7.7 us in one CTA, 6.4 in eight; over 4,096: 10.1 in eight
        and 9.6 in 32 with the merge; over 16,384: 21.8 and 11.8)."""
        return 1 if buckets <= 256 else 8 if buckets <= 4096 else 32 if rows == 1 else 16

    def _decodes_in_one_call(self, q: torch.Tensor, positions: torch.Tensor, k: torch.Tensor, v: torch.Tensor,
                             index: FlatIndex) -> bool:
        """Whether a step may go to the GPU as one call: where the calls it is made of would take these tensors as they are, and
        the methods that make them are this class's own."""
        d, b = self.design, index.buckets
        if _stages_of(type(self)) != _DECODE_STAGES or not _STAGE_NAMES.isdisjoint(self.__dict__):
            return False
        return q.dim() == 3 and 0 < q.shape[0] <= 8 and q.shape[1:] == (self.heads, self.head_dim) and d.early_budget is None \
            and index.shapes is None and d.top_p <= 128 and self.index_dim in (32, 64) and not probe.listening() \
            and positions.dtype == torch.int64 and positions.shape == q.shape[:1] and q.stride(2) == k.stride(2) == v.stride(2) == 1 \
            and k.stride() == v.stride() and k.shape[1:] == v.shape[1:] == (self.kv_heads, self.head_dim) \
            and q.dtype == k.dtype == v.dtype == torch.bfloat16 and positions.is_contiguous() \
            and b.bucket_centroids.dtype == torch.float32 and b.bucket_members.dtype == torch.int32 \
            and b.bucket_centroids.is_contiguous() and b.bucket_members.is_contiguous() \
            and b.bucket_centroids.shape[1] == self.index_dim and b.bucket_members.shape[0] == b.bucket_centroids.shape[0]

    def decode(self, q: torch.Tensor, positions: torch.Tensor, k: torch.Tensor, v: torch.Tensor, index: FlatIndex,
               splits: int = 8):
        """One step for rows at `positions` over a cache whose index is built: out [R,Hq,dh] bf16."""
        if self._decodes_in_one_call(q, positions, k, v, index):
            d, b = self.design, index.buckets
            return ops.flat_decode(q, self.query_map, self.dh_off, self.dh_used, positions, b.bucket_centroids, b.bucket_members,
                                   d.cluster_block_size, d.block_bucket_count, d.top_p, d.top_k, d.sink_size, d.window_size,
                                   self._decode_splits(q.shape[0], b.bucket_centroids.shape[0]), k, v, self.scale, splits,
                                   self._expand_status)
        lists, lengths = self.select(self.index_queries(q), positions, index)
        out, _ = self.attend(q, k, v, lists, lengths, splits=splits)
        return out


# What `FlatLayer.decode` is made of: a layer that has another of these has it called.
_STAGE_NAMES = frozenset(("index_queries", "select", "_select", "_pick", "attend"))
_stages_of = operator.attrgetter(*_STAGE_NAMES)
_DECODE_STAGES = _stages_of(FlatLayer)
