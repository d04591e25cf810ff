"""Memory that a launch or a copy in flight reads stays taken until it has: on the CPU, with the native calls replaced."""
import contextlib
import weakref

import numpy as np
import pytest
import torch


class _Lib:
    """Stands for the native library: answers the install's calls and looks at what is alive while one runs."""

    def __init__(self, seen):
        self.seen = seen

    def wa_hkv_install_table_bytes(self, *sizes):
        return 256

    def wa_hkv_install_table(self, *args):
        return 0

    def wa_hkv_install_pages_mirrored(self, job, table, rotations, mirror, stream):
        self.mirror = mirror
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
    word = torch.zeros(1, dtype=torch.int32)
    monkeypatch.setattr(_lib, "status_word", lambda dev: word)
    dst = caches.starts(1, 2)
    assert hkv._install_fused(cache, plan, dst[None], caches, dst, np.full(1, -1), None, 22, torch.device("cpu"), hsa)
    assert lib.seen == [[True]] and lib.mirror == word.data_ptr()


@pytest.mark.parametrize("call", ["store", "retrieve", "apply"])
def test_a_launch_that_gave_up_raises_in_the_next_call_of_the_bank(monkeypatch, call):
    from worldattention_b200 import _lib
    from worldattention_b200.hkv import HKVCache
    hkv = HKVCache(frame_seq_length=4, page_size_frames=2)
    k = torch.zeros(1, 8, 1, 8)
    cache = [{"k": k, "v": k.clone(), "local_end_index": torch.tensor([8]), "global_end_index": torch.tensor([8])}]
    hkv.chunks = [{"page_spans": [(0, 8)], "start_frame": 0}]
    hkv.tier.put(0, {"k": [k], "v": [k]})
    word = torch.tensor([304], dtype=torch.int32)
    monkeypatch.setitem(_lib._status_words, 0, word)
    monkeypatch.setattr(_lib, "require_cuda", lambda *t: torch.device("cuda", 0))
    on_device = type("T", (), {"is_cuda": True, "device": torch.device("cuda", 0)})()
    with pytest.raises(RuntimeError, match="HKV install.*304"):
        if call == "store":
            hkv.store(cache, prompt_embeds=k[0], current_start_frame=2, temporal_freqs=None)
        elif call == "retrieve":
            hkv.retrieve(prompt_embeds=on_device, query_vec=None)
        else:
            hkv.apply(cache, [(0, 0)], current_start_frame=2, temporal_freqs=None)
    assert int(word) == 0 and int(cache[0]["global_end_index"]) == 8


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


def test_promoted_pages_are_known_to_the_allocator_of_host_memory(monkeypatch):
    from worldattention_b200 import _lib
    from worldattention_b200.hkv import cache as C
    order, known = [], [True]

    class Side:
        stream_id, device_index, cuda_stream = 7, 0, 70
        wait_stream = lambda self, other: order.append("behind")
        synchronize = lambda self: order.append("waited for")

    class Lib:
        wa_hkv_promote_pages = lambda self, records, n, *rest: order.append(("copied", n)) or 0

    class Host:
        read_on_stream = lambda self, pages, stream_id, device: order.append(("told", [id(p) for p in pages], stream_id, device)) or known[0]
    monkeypatch.setattr(_lib, "lib", lambda: Lib())
    monkeypatch.setattr(_lib, "host", lambda: Host())
    monkeypatch.setattr(_lib, "device_guard", lambda dev: contextlib.nullcontext())
    monkeypatch.setattr(torch.cuda, "current_stream", lambda dev: None)
    monkeypatch.setattr(torch.Tensor, "record_stream", lambda t, stream: None)
    hkv = C.HKVCache(frame_seq_length=4, page_size_frames=2)
    monkeypatch.setattr(hkv.tier, "side_stream", lambda dev: Side())
    k0 = torch.zeros(2, 16, 1, 8)
    pages = [torch.zeros(2, 8, 1, 8) for _ in range(3)]
    single = [(0, "k", 0, pages[0], 0), (0, "v", 0, pages[1], None), (1, "k", 0, pages[2], 128)]
    for known[0] in (True, False):
        order.clear()
        hkv._promote(single, 256, k0)
        told = ("told", [id(pages[0]), id(pages[2])], 7, 0)
        assert order == ["behind", ("copied", 4), told] + ([] if known[0] else ["waited for"])


@pytest.mark.gpu
@pytest.mark.parametrize("tier", ["file", "host"])
def test_host_pages_are_not_handed_out_again_while_they_cross(tmp_path, tier):
    """The copies of a cold install wait behind other work; what is let go and allocated meanwhile must not reach them."""
    import worldattention_b200 as wa
    dev, frame, layers = torch.device("cuda:0"), 64, 3
    hkv = wa.hkv.HKVCache(frame_seq_length=frame, page_size_frames=2, cpu_max_chunks=1, nvme_enabled=tier == "file", nvme_dir=str(tmp_path), rerope=False)
    make = lambda n: torch.randn((1, n, 2, 128), device=dev).bfloat16()
    end = lambda: torch.tensor([4 * frame], device=dev)
    fill = lambda: [{"k": make(4 * frame), "v": make(4 * frame), "local_end_index": end(), "global_end_index": end()} for _ in range(layers)]
    freqs = torch.polar(torch.ones(64, 22, dtype=torch.float64), torch.randn(64, 22, dtype=torch.float64))
    first = fill()
    for window in (first, fill())[: 2 if tier == "file" else 1]:
        hkv.store(window, prompt_embeds=make(1).float()[:, :, 0], current_start_frame=4, temporal_freqs=freqs)
    assert hkv.tier.location(0) == ("nvme" if tier == "file" else "cpu")
    cache = fill()
    busy = torch.empty(1 << 30, dtype=torch.uint8, device=dev)
    # page-locking new memory waits for the device: what is wanted below has to be there
    buffers = lambda: [torch.full((1, n * frame, 2, 128), 7.0, dtype=torch.bfloat16, pin_memory=True) for n in (2, 4) for _ in range(4 * layers)]
    hkv.apply(fill(), [(0, 0), (0, 1)], current_start_frame=9, temporal_freqs=freqs)
    small = [torch.empty(1 << bits, dtype=torch.uint8, pin_memory=True) for bits in range(4, 17) for _ in range(8)]
    spare = buffers() + buffers()
    torch.cuda.synchronize()
    del small, spare
    with torch.cuda.stream(hkv.tier.side_stream(dev)):
        for _ in range(600):                                    # some 100 ms
            busy[: 1 << 29].copy_(busy[1 << 29:])
        done = torch.cuda.Event()
        done.record()
    assert hkv.apply(cache, [(0, 0), (0, 1)], current_start_frame=9, temporal_freqs=freqs) == 4 * frame
    if tier == "host":
        hkv.reset()
    others = buffers()
    assert not done.query(), "the copies were over before anything could reach them: this says nothing"
    torch.cuda.synchronize()
    for got, want in zip(cache, first):
        assert torch.equal(got["k"], want["k"]) and torch.equal(got["v"], want["v"])
    del others


@pytest.mark.parametrize("frame,heads,head_dim", [(218, 1, 128), (1500, 1, 128), (16, 3, 64), (16, 32, 4)])
def test_an_install_that_is_not_covered_puts_no_tables_together(monkeypatch, frame, heads, head_dim):
    from worldattention_b200.hkv import cache as C
    from worldattention_b200.hsa import HSAAttention
    hkv = C.HKVCache(frame_seq_length=frame, page_size_frames=2)
    make = lambda n: torch.zeros(1, n, heads, head_dim, dtype=torch.bfloat16)
    cache = [{"k": make(2 * frame), "v": make(2 * frame), "k_coarse": make(48), "v_coarse": make(48)}]
    caches = C._Table([cache[0]["k"], cache[0]["v"]])
    hsa = [HSAAttention(heads, head_dim, block_size=64, proj_segment_len=frame)]
    plan = np.zeros(1, dtype=hkv._PLAN_DTYPE)
    plan["count"] = 2 * frame
    monkeypatch.setattr(C, "_Table", lambda tensors: pytest.fail("put together for nothing"))
    dst = caches.starts(1, 2)
    assert hkv._install_fused(cache, plan, dst[None], caches, dst, np.full(1, -1), None, 22, torch.device("cpu"), hsa) is False
