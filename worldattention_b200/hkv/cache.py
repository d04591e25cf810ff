"""Hierarchical KV Cache (HKV) on B200 (reference: pipeline/hkv/cache.py).

The history of an autoregressive rollout is kept outside the online cache as *chunks* split into
fixed-size *pages*; a prompt switch retrieves the most relevant pages and installs exactly those
into the online cache.  Interface, page/span arithmetic, re-rotation plan and soft-failure
behaviour follow the reference.  What changes is where the bytes move:

* `store` copies the populated cache device-to-device (hot tier) or into page-locked host memory
  on a side stream, and builds the page index from layer 0's keys with one pooling kernel that
  removes the temporal rotation on the fly;
* `retrieve` scores and selects pages in one kernel launch and reads back only the chosen ids;
* `apply` installs all pages of all layers with one launch (keys re-rotated in flight, values
  verbatim), promoting host-resident pages through page-locked async copies on a side stream, and
  clears only the tail of the cache beyond the installed span.  Pages of whole frames are compressed
  by the same launch, straight into the cache slots; others by the compress kernel behind it.

Online cache contract: a list with one dict per transformer block holding `k`, `v`
(`[B, capacity, H, D]`), scalar tensors `global_end_index`, `local_end_index`, and optionally
`k_coarse`, `v_coarse`.
"""
from __future__ import annotations

import ctypes
from typing import List, Optional, Sequence, Tuple

import numpy as np
import torch

from .. import _lib
from .install import RECORD_DTYPE, clear_rows_device, gather_records_device
from .retrieval import page_key_index, prompt_index, score_and_topk, select_top_chunks
from .rope import host_table, rotation_table, temporal_complex_dims, to_device
from .tiering import HKVTierManager

__all__ = ["HKVCache"]


class _Table:
    """Addresses, sizes and strides of a list of tensors as arrays."""

    def __init__(self, tensors):
        t = np.frombuffer(_lib.host().tensor_table(tensors), dtype=np.int64).reshape(-1, 12)
        self.columns = t
        self.ptr, self.device, self.dtype, self.dim, self.size, self.stride = t[:, 0], t[:, 1], t[:, 2], t[:, 3], t[:, 4:8], t[:, 8:]

    def cache_rows(self, like: "_Table") -> np.ndarray:
        """Which tensors hold token rows of the heads, type and device of `like`'s first without gaps inside a row or between rows."""
        _, device, dtype, _, _, _, heads, head_dim = like.columns[0, :8].tolist()
        # device, type, dimensions; heads and channels; strides of rows, heads and channels
        return (self.columns[:, (1, 2, 3, 6, 7, 9, 10, 11)] == (device, dtype, 4, heads, head_dim, heads * head_dim, head_dim, 1)).all(axis=1)

    def starts(self, batch: int, esize: int) -> np.ndarray:
        """`[tensor, batch item]` addresses."""
        return self.ptr[:, None] + self.stride[:, :1] * (np.arange(batch, dtype=np.int64) * esize)


class HKVCache:
    """KV bank with two-stage page retrieval and multi-tier residency.

    Args (reference: cache.py:39-71):
        frame_seq_length: tokens per latent frame.
        page_size_frames: frames per page.
        topk_pages: page budget installed per retrieval.
        stage1_topk_chunks: how many prompt-similar chunks feed stage 2.
        cpu_max_chunks: host-resident chunk capacity.
        nvme_enabled, nvme_dir: enable and locate the NVMe tier.
        rerope: re-rotate retrieved keys to the cache slots they are replayed at.
        hbm_max_chunks: (addition) chunks kept on the GPU in front of the host tier.
    """

    def __init__(self, *, frame_seq_length: int, page_size_frames: int = 8, topk_pages: int = 4,
                 stage1_topk_chunks: int = 1, cpu_max_chunks: int = 64, nvme_enabled: bool = False,
                 nvme_dir: Optional[str] = None, rerope: bool = True, hbm_max_chunks: int = 0):
        self.frame_seq_length = int(frame_seq_length)
        self.page_size_frames = int(page_size_frames)
        self.topk_pages = int(topk_pages)
        self.stage1_topk_chunks = int(stage1_topk_chunks)
        self.rerope = bool(rerope)
        self._tier_kwargs = dict(cpu_max_chunks=cpu_max_chunks, nvme_enabled=nvme_enabled, nvme_dir=nvme_dir,
                                 hbm_max_chunks=hbm_max_chunks)
        self._table_stream: Optional[torch.cuda.Stream] = None
        self.reset()

    def reset(self) -> None:
        """Drop the bank and start a fresh rollout."""
        self.chunks: List[dict] = []
        self.prompt_bank: List[torch.Tensor] = []
        self.tier = HKVTierManager(**self._tier_kwargs)

    def __len__(self) -> int:
        return len(self.chunks)

    @property
    def page_tokens(self) -> int:
        return self.page_size_frames * self.frame_seq_length

    def _fetch_table(self, temporal_freqs):
        """The frequency table on its way to the host, on a stream that carries nothing else: a function that waits for it (and
        not for the copies launched meanwhile)."""
        if not (isinstance(temporal_freqs, torch.Tensor) and temporal_freqs.is_cuda):
            table = host_table(temporal_freqs)
            return lambda: table
        dev = temporal_freqs.device
        if self._table_stream is None or self._table_stream.device != dev:
            self._table_stream = torch.cuda.Stream(dev)
        self._table_stream.wait_stream(torch.cuda.current_stream(dev))
        with torch.cuda.stream(self._table_stream):
            landed = torch.empty(temporal_freqs.shape, dtype=temporal_freqs.dtype, pin_memory=True)
            # a lazy conjugate is resolved on the device: copy_ would do it on the host, ahead of what it does not wait for
            landed.copy_(temporal_freqs.detach().resolve_conj().resolve_neg(), non_blocking=True)
            done = torch.cuda.Event()
            done.record()
        temporal_freqs.record_stream(self._table_stream)

        def wait():
            done.synchronize()
            return landed.numpy()
        return wait

    # ------------------------------------------------------------------ store
    def store(self, kv_cache: Sequence[dict], *, prompt_embeds: torch.Tensor, current_start_frame: int,
              temporal_freqs: torch.Tensor) -> int:
        """Write the populated part of the online cache into the bank as a new chunk (cache.py:87-133).

        Returns the new chunk id, or -1 when the cache holds nothing to store.
        """
        valid_tokens = int(kv_cache[0]["local_end_index"].item())
        if valid_tokens <= 0:
            return -1
        _lib.raise_if_failed(_lib.require_cuda(kv_cache[0]["k"]))
        tensors = [block[name] for name in ("k", "v") for block in kv_cache]
        table = _Table(tensors)
        if (table.size[:, 1] < valid_tokens).any():      # the copy kernel takes addresses: nothing behind it would stop at the end of a cache
            raise RuntimeError(f"local_end_index says {valid_tokens} tokens, but an online cache tensor holds {table.size[:, 1].min()} rows")
        temporal_freqs = self._fetch_table(temporal_freqs)

        chunk_id = len(self.chunks)
        # one allocation for the whole chunk (views per layer) instead of one per layer and tensor: growing the
        # allocator's pool costs a driver call per allocation, which at 60 calls per stored window showed as stalls of
        # up to a second at a prompt switch
        first = kv_cache[0]["k"]
        uniform = bool((table.size == table.size[0]).all() and (table.dtype == table.dtype[0]).all() and (table.device == table.device[0]).all())
        blob = {"k": [], "v": []}
        if uniform:
            slab = torch.empty((2, len(kv_cache), first.shape[0], valid_tokens) + tuple(first.shape[2:]), dtype=first.dtype,
                               device=first.device)
            self._copy_rows(tensors, table, slab, valid_tokens)
            for which, name in enumerate(("k", "v")):
                blob[name] = list(slab[which])
        else:
            for block in kv_cache:
                blob["k"].append(block["k"][:, :valid_tokens].detach().clone())
                blob["v"].append(block["v"][:, :valid_tokens].detach().clone())

        page_spans = [(start, min(start + self.page_tokens, valid_tokens))
                      for start in range(0, valid_tokens, self.page_tokens)]
        start_frame = int(current_start_frame - valid_tokens // self.frame_seq_length)
        page_index = page_key_index(blob["k"][0], page_spans, frame_seq_length=self.frame_seq_length,
                                    start_frame=start_frame, temporal_freqs=temporal_freqs())
        self.chunks.append({
            "chunk_id": chunk_id,
            "valid_tokens": valid_tokens,
            "page_spans": page_spans,
            "start_frame": start_frame,
            "page_index": page_index,
            "heads": int(kv_cache[0]["k"].shape[2]),
        })
        self.prompt_bank.append(prompt_index(prompt_embeds).detach().to(page_index.device))
        self.tier.put(chunk_id, blob)
        return chunk_id

    # ------------------------------------------------------------------ retrieve
    def retrieve(self, *, prompt_embeds: torch.Tensor, query_vec: torch.Tensor,
                 per_head: bool = False):
        """Select the pages to install for the incoming prompt (cache.py:135-178).

        Returns `(chunk_id, page_id)` pairs in chronological order.  With `per_head=True` (an
        addition) the page vectors are scored per head and a list of such lists, one per head,
        is returned.
        """
        if not self.chunks:
            return []
        if prompt_embeds.is_cuda:
            _lib.raise_if_failed(prompt_embeds.device)
        bank = torch.stack(self.prompt_bank, dim=0)
        candidates = select_top_chunks(prompt_index(prompt_embeds).detach(), bank, self.stage1_topk_chunks)

        owners: List[Tuple[int, int]] = []
        vectors = []
        for chunk_id in candidates:
            page_index = self.chunks[chunk_id].get("page_index")
            if page_index is None or page_index.numel() == 0:
                continue
            vectors.append(page_index)
            owners.extend((chunk_id, page_id) for page_id in range(page_index.shape[0]))
        if not owners:
            return []
        pool = vectors[0] if len(vectors) == 1 else torch.cat(vectors, dim=0)

        query = query_vec.reshape(-1)
        if query.shape[0] != pool.shape[1]:
            raise ValueError(f"query dim {query.shape[0]} does not match page index dim {pool.shape[1]}")

        def chronological(pairs):
            return sorted(pairs, key=lambda pair: (self.chunks[pair[0]]["start_frame"],
                                                   self.chunks[pair[0]]["page_spans"][pair[1]][0]))

        if per_head:
            heads = self.chunks[owners[0][0]].get("heads", 1)
            _, ids, _ = score_and_topk(query, pool, self.topk_pages, groups=heads)
            return [chronological([owners[i] for i in row]) for row in ids.tolist()]
        if self.topk_pages <= 0:
            return []
        _, ids, _ = score_and_topk(query, pool, self.topk_pages)
        return chronological([owners[i] for i in ids[0].tolist()])

    # ------------------------------------------------------------------ apply
    def apply(self, kv_cache: Sequence[dict], selected_pairs: Sequence[Tuple[int, int]], *,
              current_start_frame: int, temporal_freqs: torch.Tensor,
              hsa_modules: Optional[Sequence] = None) -> int:
        """Install the selected pages into the online cache, replacing its contents (cache.py:180-254).

        Returns the number of tokens installed; 0 (cache untouched) when nothing resolves.  Nothing waits for the launches: one
        that gives up at a bounded wait raises in the next call of the bank or of the attention on the device, or when the
        caller runs `_lib.raise_if_failed` after its own synchronisation.
        """
        k0 = kv_cache[0]["k"]
        plan, blobs = self._install_plan(selected_pairs, capacity=int(k0.shape[1]),
                                         current_start_frame=int(current_start_frame))
        if plan is None:
            return 0
        dev = _lib.require_cuda(k0)
        _lib.raise_if_failed(dev)
        end_token = current_start_frame * self.frame_seq_length      # a float or a 0-dim tensor as well
        if isinstance(end_token, torch.Tensor):
            end_token = end_token.item()
        tokens = int(plan["count"].sum())
        if self.rerope and tokens > 0:
            temporal_freqs = self._fetch_table(temporal_freqs)

        compressed = all(name in kv_cache[0] for name in ("k_coarse", "v_coarse"))
        if compressed and hsa_modules is None:
            raise ValueError(
                "the online cache carries a compressed tier, so hsa_modules must be supplied so it "
                "can be rebuilt for the installed pages"
            )

        # Only the tails beyond the installed span and its compressed slots need clearing: the copy and compress kernels write
        # everything before them.  They go first, so that the device is at work while the copy records are put together.
        sources = self._install_sources(kv_cache, plan, blobs, k0.dtype) if tokens > 0 else None
        self._clear_tails(kv_cache, tokens, hsa_modules if compressed else None, dev)
        if tokens > 0 and not self._install(kv_cache, plan, sources, temporal_freqs, dev, k0.dtype, hsa_modules if compressed else None):
            if compressed:
                for layer, block in enumerate(kv_cache):
                    self._write_coarse(block, hsa_modules[layer], tokens)

        self._set_ends(kv_cache, "global_end_index", end_token)
        self._set_ends(kv_cache, "local_end_index", tokens)
        return tokens

    @staticmethod
    def _set_ends(kv_cache, name: str, value) -> None:
        """One index of every layer to `value`, in two launches for all layers where they can be."""
        ends = list({id(block[name]): block[name] for block in kv_cache}.values())
        if len({t.data_ptr() for t in ends}) == len(ends) and all(t.is_cuda and t.dtype == torch.long for t in ends):
            torch._foreach_zero_(ends)
            torch._foreach_add_(ends, int(value))        # which `fill_` makes of a fraction too
        else:
            for t in ends:
                t.fill_(value)

    _PLAN_DTYPE = np.dtype([("chunk", "<i8"), ("src", "<i8"), ("count", "<i8"), ("dst", "<i8"),
                            ("frame_from", "<i8"), ("frame_to", "<i8")])

    def _install_plan(self, selected_pairs, *, capacity: int, current_start_frame: int):
        """The install as a table, one row per page that resolves and (at least partly) fits.

        Columns: owning chunk, first source token and token count inside the chunk, first destination token in
        the cache, and the frame the page was written at / is replayed at.  Pairs that name an unknown chunk or
        page, or a chunk no tier holds any more, are left out (cache.py:256-271); pages fill the cache front to
        back and the one that crosses the capacity is cut (cache.py:203-211); the installed span ends at
        `current_start_frame`, so a page's new frame is that minus the frames still to come (cache.py:273-287).
        Returns `(None, {})` when no row remains.
        """
        blobs: dict = {}
        rows = []
        for chunk_id, page_id in selected_pairs:
            meta = self.chunks[chunk_id] if 0 <= chunk_id < len(self.chunks) else None
            if meta is None or not 0 <= page_id < len(meta["page_spans"]):
                continue
            if chunk_id not in blobs:
                # a spilled chunk is read page by page from its file; anything else comes as a whole blob
                held = self.tier.page_reader(chunk_id) or self.tier.get(chunk_id)
                if held is None:
                    continue
                blobs[chunk_id] = held
            first, last = meta["page_spans"][page_id]
            rows.append((chunk_id, first, last - first))
        if not rows:
            return None, {}
        plan = np.zeros(len(rows), dtype=self._PLAN_DTYPE)
        plan["chunk"], plan["src"], plan["count"] = (np.asarray(col, dtype=np.int64) for col in zip(*rows))
        before = np.cumsum(plan["count"]) - plan["count"]               # tokens installed ahead of each page
        plan["count"] = np.clip(capacity - before, 0, plan["count"])    # the page that crosses the capacity is cut
        plan = plan[: int(np.searchsorted(before, capacity, side="left"))] if capacity > 0 else plan[:0]
        if plan.size == 0:
            plan = np.zeros(1, dtype=self._PLAN_DTYPE)   # everything resolved but nothing fits: an empty install
            plan["chunk"] = rows[0][0]
        plan["dst"] = np.cumsum(plan["count"]) - plan["count"]
        frame_len = self.frame_seq_length
        chunk_frame = np.asarray([self.chunks[int(c)]["start_frame"] for c in plan["chunk"]], dtype=np.int64)
        plan["frame_from"] = chunk_frame + plan["src"] // frame_len
        plan["frame_to"] = current_start_frame - int(plan["count"].sum()) // frame_len + plan["dst"] // frame_len
        return plan, blobs

    @staticmethod
    def _copied_by_kernel(like: torch.Tensor) -> bool:
        """Whether the page-copy kernel takes rows of this type and head size."""
        return like.dtype in (torch.float32, torch.bfloat16) and like.shape[3] % 2 == 0

    @classmethod
    def _copy_rows(cls, sources, table: _Table, slab: torch.Tensor, tokens: int) -> None:
        """The first `tokens` rows of the cache tensors into `slab` `[2, layers, B, tokens, H, D]`: one launch of the page-copy
        kernel (6 GB read and written for a full window of 30 blocks: 1.75 ms against 2.05 ms as a copy per tensor)."""
        like = sources[0]
        rows = slab.view(-1, *slab.shape[2:])
        if not (cls._copied_by_kernel(like) and table.cache_rows(table).all()):
            for dst, t in zip(rows, sources):
                dst.copy_(t[:, :tokens].detach())
            return
        records = np.zeros((len(sources), like.shape[0]), dtype=RECORD_DTYPE)
        row_elems, esize = like.shape[2] * like.shape[3], like.element_size()
        items = np.arange(len(sources) * like.shape[0], dtype=np.int64).reshape(records.shape)
        records["src"] = table.starts(like.shape[0], esize).astype(np.uint64)
        records["dst"] = (slab.data_ptr() + items * (tokens * row_elems * esize)).astype(np.uint64)
        records["src_stride"] = records["dst_stride"] = row_elems
        records["n_tokens"], records["rot"] = tokens, -1
        gather_records_device(to_device(records.reshape(-1).view(np.uint8), like.device), max_tokens=tokens, row_elems=row_elems,
                              head_dim=like.shape[3], dtype=like.dtype)

    @classmethod
    def _clear_tails(cls, kv_cache, tokens: int, hsa_modules, dev) -> None:
        """Zero everything behind the installed tokens (and, with `hsa_modules`, behind their compressed slots) in all
        layers in one launch."""
        k0 = kv_cache[0]["k"]
        row_elems, esize = k0.shape[2] * k0.shape[3], k0.element_size()
        tensors, ends = [], []
        for layer, block in enumerate(kv_cache):
            tensors += [block["k"], block["v"]]
            ends += [tokens, tokens]
            if hsa_modules is not None:
                slots = hsa_modules[layer].token_range_to_coarse(0, tokens)[1] if tokens > 0 else 0
                tensors += [block["k_coarse"], block["v_coarse"]]
                ends += [slots, slots]
        table, ends = _Table(tensors), np.array(ends, dtype=np.int64)
        rows = table.size[:, 1] - ends
        direct = table.cache_rows(table) if cls._copied_by_kernel(k0) else np.zeros(len(rows), dtype=bool)
        for i in np.flatnonzero((rows > 0) & ~direct):
            tensors[i][:, int(ends[i]):].zero_()
        mine = np.flatnonzero((rows > 0) & direct)
        if mine.size == 0:
            return
        items, batch = mine, 0                                                           # a record per tensor and batch item
        if (table.size[mine, 0] != 1).any():
            items, batch = np.repeat(mine, table.size[mine, 0]), np.concatenate([np.arange(n) for n in table.size[mine, 0]])
        records = np.zeros(len(items), dtype=RECORD_DTYPE)
        records["dst"] = (table.ptr[items] + (batch * table.stride[items, 0] + ends[items] * row_elems) * esize).astype(np.uint64)
        records["n_tokens"], records["dst_stride"] = rows[items], row_elems
        clear_rows_device(to_device(records.view(np.uint8), dev), max_tokens=int(rows[mine].max()), row_elems=row_elems, elem_size=esize)

    def _install_sources(self, kv_cache, plan, blobs, dtype):
        """Where the pages come from and go to: `(whole, single, staging, caches)`; cold pages are on their way to the staging buffer.

        `whole` maps a chunk that lies on the device in the cache's own layout to the tensors of all layers and their table (its
        pages are rows of those); `single` lists the pages of every other chunk one by one, as (layer, name, plan row, tensor or host
        page, offset in the staging buffer or None); `caches` is the table of the online tensors, (layer, K|V).
        """
        k0 = kv_cache[0]["k"]
        bsz, _, heads, head_dim = k0.shape
        row_elems = heads * head_dim
        _lib.dtype_code(dtype)               # raises for a type that the page-copy kernel does not take
        caches = _Table([block[name] for block in kv_cache for name in ("k", "v")])
        if (caches.stride[:, 1:] != (row_elems, head_dim, 1)).any():
            raise ValueError("online cache tensors must be contiguous [B, capacity, H, D]")
        whole = {}
        for chunk_id, held in blobs.items():
            if not callable(held):
                tensors = [held[name][layer] for layer in range(len(kv_cache)) for name in ("k", "v")]
                table = _Table(tensors)
                if table.cache_rows(caches).all() and (table.size[:, 0] == bsz).all():
                    whole[chunk_id] = (tensors, table)
        single, staged_elems = [], 0
        rows = [(i, int(row["chunk"]), int(row["src"]), int(row["count"])) for i, row in enumerate(plan)]
        rows = [row for row in rows if row[3] and row[1] not in whole]
        for layer in range(len(kv_cache) if rows else 0):
            for name in ("k", "v"):
                for i, chunk_id, first, n in rows:
                    held = blobs[chunk_id]
                    page = held(name, layer, first, first + n) if callable(held) else held[name][layer][:, first: first + n]
                    slot = None
                    if not page.is_cuda and page.dtype == dtype and page.stride(3) == 1 and page.stride(2) == head_dim \
                            and page.stride(1) == row_elems:
                        slot = staged_elems                      # cold page in the cache's own layout: one block copy per item
                        staged_elems += bsz * n * row_elems
                    single.append((layer, name, i, page, slot))
        return whole, single, self._promote(single, staged_elems, k0) if staged_elems else None, caches

    def _promote(self, single, staged_elems: int, k0: torch.Tensor) -> torch.Tensor:
        """Cold pages in the cache's own layout cross on the side stream into ONE staging buffer, one block copy per item: the first
        thing that is launched, since the link is what a cold install waits for."""
        dev = k0.device
        bsz, _, heads, head_dim = k0.shape
        row_elems, esize = heads * head_dim, k0.element_size()
        staging = torch.empty((staged_elems,), dtype=k0.dtype, device=dev)
        promote = []
        for _, _, _, page, slot in single:
            if slot is not None:
                n = page.shape[1]
                promote += [_lib.PageCopy(page.data_ptr() + b * page.stride(0) * esize, staging.data_ptr() + (slot + b * n * row_elems) * esize,
                                          row_elems, row_elems, n, -1) for b in range(bsz)]
        main, side = torch.cuda.current_stream(dev), self.tier.side_stream(dev)
        side.wait_stream(main)            # the staging block may be recycled memory that the main stream still uses
        staging.record_stream(side)
        try:
            with _lib.device_guard(dev):
                _lib.check(_lib.lib().wa_hkv_promote_pages((_lib.PageCopy * len(promote))(*promote), len(promote), row_elems, esize, side.cuda_stream))
        finally:
            # nobody waits here, and a page read from a file is dropped as soon as the install is enqueued, a chunk's when the bank
            # lets go of it: their page-locked memory must not be handed out again before the copies are done
            if not _lib.host().read_on_stream([page for _, _, _, page, slot in single if slot is not None], side.stream_id, side.device_index):
                side.synchronize()
        return staging

    def _install(self, kv_cache, plan, sources, temporal_freqs, dev, dtype, hsa_modules=None) -> bool:
        """The plan's pages into the caches of all layers in one launch.

        With `hsa_modules` and where the fused kernel covers the call, the compressed slots are written by that launch too
        (True); otherwise one page-copy launch for every (layer, page, K|V, batch item) (False)."""
        whole, single, staging, caches = sources
        k0 = kv_cache[0]["k"]
        bsz, _, heads, head_dim = k0.shape
        row_elems = heads * head_dim
        esize = k0.element_size()
        nt = temporal_complex_dims(head_dim)
        rot = None
        if self.rerope:
            rot = rotation_table(temporal_freqs(), plan["frame_to"].tolist(), plan["frame_from"].tolist(), nt)

        main = torch.cuda.current_stream(dev)
        side = self.tier.side_stream(dev)
        # whatever conversion a cold page needs runs on the side stream too, behind its copy, so that nothing reads a landing
        # buffer early
        keep_alive = [staging]
        promoted = staging is not None
        # first row of every (page, tensor, batch item) on the device, elements between its rows
        dst = caches.starts(bsz, esize)
        batch = np.arange(bsz, dtype=np.int64) * esize
        src = np.zeros((len(plan),) + dst.shape, dtype=np.int64)
        src_stride = np.full(src.shape[:2], row_elems, dtype=np.int64)
        for layer, name, i, page, slot in single:
            row = plan[i]
            n = int(row["count"])
            if slot is not None:
                src_ptr, src_batch, stride = staging.data_ptr() + slot * esize, n * row_elems, row_elems
            else:
                if not page.is_cuda:
                    with torch.cuda.stream(side):
                        landed = torch.empty(page.shape, dtype=page.dtype, device=dev)
                        landed.copy_(page, non_blocking=True)
                        page = self._as_cache_rows(landed, dtype, head_dim)
                    promoted = True
                else:
                    page = self._as_cache_rows(page, dtype, head_dim)
                keep_alive.append(page)
                src_ptr, src_batch, stride = page.data_ptr(), page.stride(0), page.stride(1)
            at = 2 * layer + (name == "v")
            src[i, at] = src_ptr + batch * src_batch
            src_stride[i, at] = stride
        for chunk_id, (_, table) in whole.items():
            mine = np.flatnonzero(plan["chunk"] == chunk_id)
            src[mine] = table.starts(bsz, esize) + (plan["src"][mine] * (row_elems * esize))[:, None, None]
        if promoted:
            main.wait_stream(side)
        used = np.flatnonzero(plan["count"] > 0)
        rot_dev = to_device(rot, dev) if rot is not None else None
        fused = hsa_modules is not None and bool((src_stride[used] == row_elems).all()) and self._install_fused(
            kv_cache, plan[used], src[used], caches, dst, used if rot is not None else np.full(len(used), -1), rot_dev, nt, dev, hsa_modules)
        if not fused:
            records = np.zeros((len(used),) + dst.shape, dtype=RECORD_DTYPE)
            records["src"] = src[used].astype(np.uint64)
            records["dst"] = (dst + (plan["dst"][used] * (row_elems * esize))[:, None, None]).astype(np.uint64)
            records["src_stride"], records["dst_stride"] = src_stride[used][:, :, None], row_elems
            records["n_tokens"] = plan["count"][used][:, None, None]
            records["rot"] = -1
            if rot is not None:
                records["rot"][:, ::2] = used[:, None, None]
            gather_records_device(to_device(records.reshape(-1).view(np.uint8), dev), max_tokens=int(plan["count"].max()), row_elems=row_elems,
                                  head_dim=head_dim, dtype=dtype, rotations=rot_dev, n_temporal=nt)
        storages = {t.untyped_storage().data_ptr(): t for t in keep_alive if t is not None and t.is_cuda}
        for held, _ in whole.values():
            storages.update((t.untyped_storage().data_ptr(), t) for t in held)
        for t in storages.values():
            t.record_stream(main)
        return fused

    def _install_fused(self, kv_cache, plan, src, caches, dst, rot_rows, rot_dev, nt, dev, hsa_modules) -> bool:
        """Copy, rotation and compression of all layers in one launch: bf16, pages of whole frames, projection segments of one
        frame, one shape of projection for all layers.  False (nothing launched): not covered."""
        k0 = kv_cache[0]["k"]
        bsz, _, heads, head_dim = k0.shape
        frame, esize = self.frame_seq_length, k0.element_size()
        # most of what the native call would refuse, before the tables that it looks at are put together (a projection of 218 or 1500
        # tokens: 150 us of host work for nothing)
        proj = getattr(hsa_modules[0], "k_proj_mat", None)
        if (k0.dtype != torch.bfloat16 or heads * head_dim % 128 or head_dim % 8 or not isinstance(proj, torch.Tensor) or proj.dim() != 2
                or proj.shape[1] % 8 or proj.dtype != k0.dtype or (plan["count"] % frame).any() or (plan["src"] % frame).any()):
            return False
        # tiers whose slots the compress kernel does not write either are the module's own business (`compress_kv_cache`), and all
        # that is asked of such a module
        coarse = _Table([layer[name] for layer in kv_cache for name in ("k_coarse", "v_coarse")])
        if not ((coarse.dim == 4).all() and (coarse.dtype == caches.dtype[0]).all() and (coarse.device == caches.device[0]).all()
                and (coarse.stride[::2] == coarse.stride[1::2]).all() and (coarse.size[:, 0] >= bsz).all()
                and (coarse.size[:, 2:] == (heads, head_dim)).all() and (coarse.stride[:, 2:] == (head_dim, 1)).all()):
            return False
        hsa_modules = [hsa_modules[layer] for layer in range(len(kv_cache))]
        first = hsa_modules[0]
        shape, block = first.k_proj_mat.shape, first.block_size
        if first.proj_segment_len != frame or shape[1] < frame or any(hsa.proj_segment_len != frame or hsa.block_size != block for hsa in hsa_modules):
            return False
        slots = first.token_range_to_coarse(0, int(plan["count"].sum()))[1]
        proj = _Table([p for hsa in hsa_modules for p in (hsa.k_proj_mat, hsa.v_proj_mat)])
        if not ((caches.dtype == caches.dtype[0]).all() and (caches.size[:, 0] == bsz).all() and (coarse.size[:, 1] >= slots).all()
                and (proj.dim == 2).all() and (proj.dtype == caches.dtype[0]).all() and (proj.device == caches.device[0]).all()
                and (proj.size[:, :2] == shape).all() and (proj.stride[:, :2] == (shape[1], 1)).all()):
            return False
        between = lambda a: np.ascontiguousarray((a[..., 1] - a[..., 0]) // esize if bsz > 1 else np.zeros(a.shape[:-1], dtype=np.int64))
        whole = lambda a: np.ascontiguousarray(a)
        frames = (plan["count"] // frame).astype(np.int32)
        arrays = dict(page_frames=frames, page_rot=rot_rows.astype(np.int32), src=np.ascontiguousarray(src[..., 0]).astype(np.uint64),
                      src_batch=between(src), dst=dst[:, 0].astype(np.uint64), dst_batch=between(dst), coarse=coarse.ptr.astype(np.uint64),
                      coarse_batch=whole(coarse.stride[:, 0]), coarse_row=whole(coarse.stride[:, 1]), proj=proj.ptr.astype(np.uint64))
        job = _lib.HkvInstall(len(plan), len(dst), int(frames.sum()), bsz, heads, head_dim, frame, block, shape[0], shape[1],
                              nt if rot_dev is not None else 0, *(arrays[n].ctypes.data for n, _ in _lib.HkvInstall._fields_[11:]))
        lib = _lib.lib()
        table = np.empty((lib.wa_hkv_install_table_bytes(job.pages, job.tensors, job.segments),), dtype=np.uint8)
        with _lib.device_guard(dev):
            rc = lib.wa_hkv_install_table(ctypes.byref(job), table.ctypes.data, table.nbytes)
            if rc == _lib.WA_ERR_UNSUPPORTED:
                return False
            _lib.check(rc)
            maps = to_device(table, dev)         # held until the launch is enqueued: its memory then stays ahead of whoever takes it next
            _lib.check(lib.wa_hkv_install_pages_mirrored(ctypes.byref(job), maps.data_ptr(), _lib.ptr(rot_dev), _lib.status_word(dev).data_ptr(),
                                                         _lib.stream_ptr(dev)))
        return True

    @staticmethod
    def _as_cache_rows(page: torch.Tensor, dtype: torch.dtype, head_dim: int) -> torch.Tensor:
        """`page` in the cache's dtype with head rows contiguous (a no-op for pages stored the way the cache is)."""
        if page.dtype != dtype:
            page = page.to(dtype)
        if page.stride(3) != 1 or page.stride(2) != head_dim:
            page = page.contiguous()
        return page

    @staticmethod
    def _write_coarse(block: dict, hsa, total_tokens: int) -> int:
        """Rebuild the compressed tier from the tokens installed at cache offset 0 (cache.py:289-299).

        The compress kernel writes directly into the cache's compressed slots.
        """
        k, v = block["k"][:, :total_tokens], block["v"][:, :total_tokens]
        dev = k.device
        bsz, _, heads, head_dim = k.shape
        coarse_start, coarse_end = hsa.token_range_to_coarse(0, int(total_tokens))
        kc, vc = block["k_coarse"], block["v_coarse"]
        if kc.dtype != k.dtype or vc.dtype != k.dtype or kc.stride() != vc.stride() or kc.stride(3) != 1:
            k_new, v_new = hsa.compress_kv_cache(k, v)
            kc[:, coarse_start:coarse_end] = k_new.to(kc.dtype)
            vc[:, coarse_start:coarse_end] = v_new.to(vc.dtype)
            return coarse_end
        if coarse_end > kc.shape[1]:
            raise ValueError("compressed cache is too small for the installed pages")
        pk = hsa.k_proj_mat.detach().to(device=dev).contiguous()
        pv = hsa.v_proj_mat.detach().to(device=dev, dtype=pk.dtype).contiguous()
        _lib.check(_lib.lib().wa_compress_kv(
            _lib.t4_blhd(k), _lib.t4_blhd(v), _lib.t4_blhd(kc), _lib.t4_blhd(vc), bsz, int(total_tokens), heads,
            head_dim, hsa.proj_segment_len, hsa.block_size, pk.data_ptr(), pv.data_ptr(), _lib.dtype_code(pk.dtype),
            pk.shape[0], pk.shape[1], _lib.stream_ptr(dev)))
        return coarse_end
