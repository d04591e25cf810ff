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

    # ------------------------------------------------------------------ store
    def store(self, kv_cache: Sequence[dict], *, prompt_embeds: torch.Tensor, current_start_frame: int,
              temporal_freqs: torch.Tensor) -> int:
        """Write the populated part of the online cache into the bank as a new chunk (cache.py:87-133).

        Returns the new chunk id, or -1 when the cache holds nothing to store.
        """
        valid_tokens = int(kv_cache[0]["local_end_index"].item())
        if valid_tokens <= 0:
            return -1
        _lib.require_cuda(kv_cache[0]["k"])
        short = next((block[name] for block in kv_cache for name in ("k", "v") if block[name].shape[1] < valid_tokens), None)
        if short is not None:          # the copy kernel takes addresses: nothing behind it would stop at the end of a cache
            raise RuntimeError(f"local_end_index says {valid_tokens} tokens, but an online cache tensor holds {short.shape[1]} rows")
        temporal_freqs = host_table(temporal_freqs)     # before the copies: it waits for the device

        chunk_id = len(self.chunks)
        # one allocation for the whole chunk (views per layer) instead of one per layer and tensor: growing the
        # allocator's pool costs a driver call per allocation, which at 60 calls per stored window showed as stalls of
        # up to a second at a prompt switch
        first = kv_cache[0]["k"]
        uniform = all(block[name].shape == first.shape and block[name].dtype == first.dtype and block[name].device == first.device
                      for block in kv_cache for name in ("k", "v"))
        blob = {"k": [], "v": []}
        if uniform:
            slab = torch.empty((2, len(kv_cache), first.shape[0], valid_tokens) + tuple(first.shape[2:]), dtype=first.dtype,
                               device=first.device)
            self._copy_rows([block[name] for name in ("k", "v") for block in kv_cache], slab, valid_tokens)
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
                                    start_frame=start_frame, temporal_freqs=temporal_freqs)
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

        Returns the number of tokens installed; 0 (cache untouched) when nothing resolves.
        """
        k0 = kv_cache[0]["k"]
        plan, blobs = self._install_plan(selected_pairs, capacity=int(k0.shape[1]),
                                         current_start_frame=int(current_start_frame))
        if plan is None:
            return 0
        dev = _lib.require_cuda(k0)
        tokens = int(plan["count"].sum())
        if self.rerope and tokens > 0:
            temporal_freqs = host_table(temporal_freqs)     # before anything is launched: it waits for the device

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

        for name, value in (("global_end_index", current_start_frame * self.frame_seq_length), ("local_end_index", tokens)):
            ends = list({id(block[name]): block[name] for block in kv_cache}.values())
            if len({t.data_ptr() for t in ends}) == len(ends) and all(t.is_cuda and t.dtype == torch.long for t in ends):
                torch._foreach_zero_(ends)           # two launches for all layers
                torch._foreach_add_(ends, value)
            else:
                for t in ends:
                    t.fill_(value)
        return tokens

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
    def _cache_rows(t: torch.Tensor, like: torch.Tensor) -> bool:
        """Whether `t` holds token rows of `like`'s heads, type and device without gaps inside a row or between rows."""
        heads, head_dim = like.shape[2:]
        return (t.dtype == like.dtype and t.device == like.device and t.shape[2:] == like.shape[2:] and t.stride(3) == 1
                and t.stride(2) == head_dim and t.stride(1) == heads * head_dim)

    @staticmethod
    def _copied_by_kernel(like: torch.Tensor) -> bool:
        """Whether the page-copy kernel takes rows of this type and head size."""
        return like.dtype in (torch.float32, torch.bfloat16) and like.shape[3] % 2 == 0

    @classmethod
    def _copy_rows(cls, sources, slab: torch.Tensor, tokens: int) -> None:
        """The first `tokens` rows of the cache tensors into `slab` `[2, layers, B, tokens, H, D]`: one launch of the page-copy
        kernel (6 GB read and written for a full window of 30 blocks: 1.75 ms against 2.05 ms as a copy per tensor)."""
        like = sources[0]
        rows = list(slab.view(-1, *slab.shape[2:]))
        if not (cls._copied_by_kernel(like) and all(cls._cache_rows(t, like) for t in sources)):
            for dst, t in zip(rows, sources):
                dst.copy_(t[:, :tokens].detach())
            return
        records = np.zeros((len(rows), like.shape[0]), dtype=RECORD_DTYPE)
        batch = np.arange(like.shape[0], dtype=np.int64) * like.element_size()
        for name, tensors in (("src", sources), ("dst", rows)):
            base, step = (np.array(x, dtype=np.int64)[:, None] for x in ([t.data_ptr() for t in tensors], [t.stride(0) for t in tensors]))
            records[name] = (base + step * batch).astype(np.uint64)
        row_elems = like.shape[2] * like.shape[3]
        records["src_stride"] = records["dst_stride"] = row_elems
        records["n_tokens"], records["rot"] = tokens, -1
        gather_records_device(to_device(records.reshape(-1).view(np.uint8), like.device), max_tokens=tokens, row_elems=row_elems,
                              head_dim=like.shape[3], dtype=like.dtype)

    @classmethod
    def _clear_tails(cls, kv_cache, tokens: int, hsa_modules, dev) -> None:
        """Zero everything behind the installed tokens (and, with `hsa_modules`, behind their compressed slots) in all
        layers in one launch."""
        k0 = kv_cache[0]["k"]
        row_elems = k0.shape[2] * k0.shape[3]
        direct = cls._copied_by_kernel(k0)
        dst, count = [], []
        for layer, block in enumerate(kv_cache):
            ends = {"k": tokens, "v": tokens}
            if hsa_modules is not None:
                slots = hsa_modules[layer].token_range_to_coarse(0, tokens)[1] if tokens > 0 else 0
                ends.update(k_coarse=slots, v_coarse=slots)
            for name, end in ends.items():
                t = block[name]
                rows = t.shape[1] - end
                if rows <= 0:
                    continue
                if not direct or not cls._cache_rows(t, k0):
                    t[:, end:].zero_()
                    continue
                for b in range(t.shape[0]):
                    dst.append(t.data_ptr() + (b * t.stride(0) + end * row_elems) * t.element_size())
                    count.append(rows)
        if not dst:
            return
        records = np.zeros(len(dst), dtype=RECORD_DTYPE)
        records["dst"], records["n_tokens"] = dst, count
        records["dst_stride"] = row_elems
        clear_rows_device(to_device(records.view(np.uint8), dev), max_tokens=max(count), row_elems=row_elems, elem_size=k0.element_size())

    def _install_sources(self, kv_cache, plan, blobs, dtype):
        """Where the pages come from: `(whole, single, staged_elems)`.

        `whole` maps a chunk that lies on the device in the cache's own layout to the tensors of all layers (its pages are
        rows of those); `single` lists the pages of every other chunk one by one, as (layer, name, plan row, tensor or host
        page, offset in the staging buffer or None), and `staged_elems` is that buffer's size.
        """
        k0 = kv_cache[0]["k"]
        bsz, _, heads, head_dim = k0.shape
        row_elems = heads * head_dim
        _lib.dtype_code(dtype)               # raises for a type that the page-copy kernel does not take
        for block in kv_cache:
            for name in ("k", "v"):
                dst = block[name]
                if dst.stride(3) != 1 or dst.stride(2) != head_dim or dst.stride(1) != row_elems:
                    raise ValueError("online cache tensors must be contiguous [B, capacity, H, D]")
        whole = {}
        for chunk_id, held in blobs.items():
            if not callable(held):
                tensors = [held[name][layer] for layer in range(len(kv_cache)) for name in ("k", "v")]
                if all(self._cache_rows(t, k0) and t.dtype == dtype and t.shape[0] == bsz for t in tensors):
                    whole[chunk_id] = tensors
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
        return whole, single, staged_elems

    def _install(self, kv_cache, plan, sources, temporal_freqs, dev, dtype, hsa_modules=None) -> bool:
        """The plan's pages into the caches of all layers in one launch.

        With `hsa_modules` and where the fused kernel covers the call, the compressed slots are written by that launch too
        (True); otherwise one page-copy launch for every (layer, page, K|V, batch item) (False)."""
        whole, single, staged_elems = sources
        k0 = kv_cache[0]["k"]
        bsz, _, heads, head_dim = k0.shape
        row_elems = heads * head_dim
        esize = k0.element_size()
        nt = temporal_complex_dims(head_dim)
        rot = None
        if self.rerope:
            rot = rotation_table(temporal_freqs, plan["frame_to"].tolist(), plan["frame_from"].tolist(), nt)

        main = torch.cuda.current_stream(dev)
        side = self.tier.side_stream(dev)
        # cold pages cross on the side stream into ONE staging buffer; whatever conversion a page needs runs on that stream too,
        # behind its copy, so that nothing reads a landing buffer early
        staging = torch.empty((max(staged_elems, 1),), dtype=dtype, device=dev) if staged_elems else None
        keep_alive = [staging]
        promote = []
        promoted = False
        # first row of every (page, tensor, batch item) on the device, elements between its rows; a tensor is (layer, K|V)
        tensors = [block[name] for block in kv_cache for name in ("k", "v")]
        batch = np.arange(bsz, dtype=np.int64) * esize
        starts = lambda ts: (np.array([t.data_ptr() for t in ts], dtype=np.int64)[:, None]
                             + np.array([t.stride(0) for t in ts], dtype=np.int64)[:, None] * batch)
        src = np.zeros((len(plan), len(tensors), bsz), dtype=np.int64)
        src_stride = np.full((len(plan), len(tensors)), row_elems, dtype=np.int64)
        for layer, name, i, page, slot in single:
            row = plan[i]
            n = int(row["count"])
            if slot is not None:
                src_ptr, src_batch, stride = staging.data_ptr() + slot * esize, n * row_elems, row_elems
                for b in range(bsz):
                    promote.append(_lib.PageCopy(page.data_ptr() + b * page.stride(0) * esize,
                                                 src_ptr + b * src_batch * esize, row_elems, row_elems, n, -1))
                keep_alive.append(page)
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
        for chunk_id, held in whole.items():
            mine = np.flatnonzero(plan["chunk"] == chunk_id)
            src[mine] = starts(held) + (plan["src"][mine] * (row_elems * esize))[:, None, None]
        if promote:
            arr = (_lib.PageCopy * len(promote))(*promote)
            side.wait_stream(main)            # the staging block may be recycled memory that the main stream still uses
            staging.record_stream(side)
            with _lib.device_guard(dev):
                _lib.check(_lib.lib().wa_hkv_promote_pages(arr, len(promote), row_elems, esize, side.cuda_stream))
            promoted = True
        if promoted:
            main.wait_stream(side)
        used = np.flatnonzero(plan["count"] > 0)
        dst = starts(tensors)
        rot_dev = to_device(rot, dev) if rot is not None else None
        fused = hsa_modules is not None and bool((src_stride[used] == row_elems).all()) and self._install_fused(
            kv_cache, plan[used], src[used], dst, used if rot is not None else np.full(len(used), -1), rot_dev, nt, dev, hsa_modules)
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
        for held in whole.values():
            storages.update((t.untyped_storage().data_ptr(), t) for t in held)
        for t in storages.values():
            t.record_stream(main)
        return fused

    def _install_fused(self, kv_cache, plan, src, dst, rot_rows, rot_dev, nt, dev, hsa_modules) -> bool:
        """Copy, rotation and compression of all layers in one launch: bf16, pages of whole frames, projection segments of one
        frame, one shape of projection for all layers.  False (nothing launched): not covered."""
        k0 = kv_cache[0]["k"]
        bsz, _, heads, head_dim = k0.shape
        frame, esize = self.frame_seq_length, k0.element_size()
        if k0.dtype != torch.bfloat16 or (plan["count"] % frame).any() or (plan["src"] % frame).any():
            return False
        first = hsa_modules[0]
        shape, block = first.k_proj_mat.shape, first.block_size
        if first.proj_segment_len != frame or shape[1] < frame:
            return False
        slots = first.token_range_to_coarse(0, int(plan["count"].sum()))[1]
        coarse, proj = [], []
        for layer, hsa in zip(kv_cache, hsa_modules):
            kc, vc = layer["k_coarse"], layer["v_coarse"]
            if hsa.proj_segment_len != frame or hsa.block_size != block or kc.stride() != vc.stride():
                return False
            for cache, t, p in ((layer["k"], kc, hsa.k_proj_mat), (layer["v"], vc, hsa.v_proj_mat)):
                if (cache.dtype != torch.bfloat16 or cache.shape[0] != bsz or t.dtype != torch.bfloat16 or p.dtype != torch.bfloat16
                        or t.device != dev or p.device != dev or p.shape != shape or not p.is_contiguous() or t.shape[0] < bsz
                        or t.shape[1] < slots or t.shape[2:] != k0.shape[2:] or t.stride(3) != 1 or t.stride(2) != head_dim):
                    return False
                coarse.append(t)
                proj.append(p)
        address = lambda ts: np.array([t.data_ptr() for t in ts], dtype=np.uint64)
        step = lambda ts, dim: np.array([t.stride(dim) for t in ts], dtype=np.int64)
        between = lambda a: np.ascontiguousarray((a[..., 1] - a[..., 0]) // esize if bsz > 1 else np.zeros(a.shape[:-1], dtype=np.int64))
        frames = (plan["count"] // frame).astype(np.int32)
        arrays = dict(page_frames=frames, page_rot=rot_rows.astype(np.int32), src=np.ascontiguousarray(src[..., 0]).astype(np.uint64),
                      src_batch=between(src), dst=dst[:, 0].astype(np.uint64), dst_batch=between(dst), coarse=address(coarse),
                      coarse_batch=step(coarse, 0), coarse_row=step(coarse, 1), proj=address(proj))
        job = _lib.HkvInstall(len(plan), len(dst), int(frames.sum()), bsz, heads, head_dim, frame, block, shape[0], shape[1],
                              nt if rot_dev is not None else 0, *(arrays[n].ctypes.data for n, _ in _lib.HkvInstall._fields_[11:]))
        lib = _lib.lib()
        table = np.empty((lib.wa_hkv_install_table_bytes(job.pages, job.tensors, job.segments),), dtype=np.uint8)
        with _lib.device_guard(dev):
            rc = lib.wa_hkv_install_table(ctypes.byref(job), table.ctypes.data, table.nbytes)
            if rc == _lib.WA_ERR_UNSUPPORTED:
                return False
            _lib.check(rc)
            _lib.check(lib.wa_hkv_install_pages(ctypes.byref(job), to_device(table, dev).data_ptr(), _lib.ptr(rot_dev), _lib.stream_ptr(dev)))
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
