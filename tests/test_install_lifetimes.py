"""Memory that a launch or a copy in flight reads stays taken until it has: on the CPU, with the native calls replaced."""
import contextlib
import weakref

import numpy as np
import torch


class _Lib:
    """Stands for the native library: answers the install's calls and looks at what is alive while one runs."""

    def __init__(self, seen):
        self.seen = seen

    def wa_hkv_install_table_bytes(self, *sizes):
        return 256

    def wa_hkv_install_table(self, *args):
        return 0

    def wa_hkv_install_pages(self, job, table, *args):
        self.seen.append([ref() is not None and ref().data_ptr() == table for ref in self.refs])
        return 0


def test_the_install_holds_its_table_while_it_launches(monkeypatch):
    from worldattention_b200 import _lib
    from worldattention_b200.hkv import cache as C
    from worldattention_b200.hsa import HSAAttention
    _lib.host()
    frame, heads, d = 16, 1, 128
    hkv = C.HKVCache(frame_seq_length=frame, page_size_frames=2)
    hsa = [HSAAttention(heads, d, block_size=64, proj_segment_len=frame) for _ in range(2)]
    make = lambda n: torch.zeros(1, n, heads, d, dtype=torch.bfloat16)
    cache = [{"k": make(80), "v": make(80), "k_coarse": make(5), "v_coarse": make(5)} for _ in range(2)]
    caches = C._Table([b[n] for b in cache for n in ("k", "v")])
    plan = np.zeros(1, dtype=hkv._PLAN_DTYPE)
    plan["count"] = 32
    lib = _Lib([])
    lib.refs = []

    def to_device(array, dev):
        t = torch.from_numpy(array).clone()
        lib.refs.append(weakref.ref(t))
        return t
    monkeypatch.setattr(C, "to_device", to_device)
    monkeypatch.setattr(_lib, "lib", lambda: lib)
    monkeypatch.setattr(_lib, "device_guard", lambda dev: contextlib.nullcontext())
    monkeypatch.setattr(_lib, "stream_ptr", lambda dev: 0)
    dst = caches.starts(1, 2)
    assert hkv._install_fused(cache, plan, dst[None], caches, dst, np.full(1, -1), None, 22, torch.device("cpu"), hsa)
    assert lib.seen == [[True]]


def test_candidates_of_a_shard_hold_their_contiguous_inputs(monkeypatch):
    from worldattention_b200 import _lib, sharded
    made, seen = [], []
    contiguous = torch.Tensor.contiguous

    def copy(t, *a):
        out = contiguous(t, *a)
        made.append(weakref.ref(out))
        return out

    class Lib:
        def call(self, *args):
            seen.append([ref() is not None for ref in made])
            return 0
        wa_route_local_candidates = wa_route_merge_candidates = call
    monkeypatch.setattr(torch.Tensor, "contiguous", copy)
    monkeypatch.setattr(_lib, "lib", lambda: Lib())
    monkeypatch.setattr(_lib, "require_cuda", lambda *t: torch.device("cpu"))
    monkeypatch.setattr(_lib, "stream_ptr", lambda dev: 0)
    sharded.local_candidates(torch.zeros(1, 3, 2, 8).transpose(1, 2), torch.zeros(1, 5, 2, 8).transpose(1, 2), block_lo=0, topk_max=2)
    made.clear()
    sharded.merge_candidates(torch.zeros(6, 2, 2, dtype=torch.int64).transpose(0, 1), (1, 2, 3), topk_per_head=torch.ones(2), blocks_total=9,
                             block_lo=0, block_hi=5)
    assert seen == [[True, True], [True, True]]
