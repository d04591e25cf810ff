"""The fused install (copy, rotation and compression of all layers in one launch) against the page-copy and compress kernels it
stands in for: the same bits, over frames of whole tiles and of remainders, batches, head sizes, tiers and unequal pages."""
import numpy as np
import pytest
import torch

from tests.helpers import dev

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("frame,heads,d,bsz,block,hot,rerope", [
    (24, 2, 64, 1, 64, 2, True), (128, 1, 128, 2, 64, 2, True), (136, 3, 128, 1, 64, 0, True), (1560, 2, 128, 1, 128, 2, True),
    (256, 4, 32, 2, 64, 1, True), (264, 2, 64, 3, 128, 2, False), (8, 1, 128, 1, 64, 2, True)])
def test_fused_install_equals_the_separate_kernels(monkeypatch, frame, heads, d, bsz, block, hot, rerope):
    import worldattention_b200 as wa
    layers, window = 3, 7
    g = torch.Generator(device=dev()).manual_seed(frame)
    make = lambda n: torch.randn((bsz, n, heads, d), generator=g, device=dev()).bfloat16()
    hsa = [wa.hsa.HSAAttention(heads, d, block_size=block, proj_segment_len=frame).to(dev(), torch.bfloat16) for _ in range(layers)]
    for m in hsa:
        torch.nn.init.normal_(m.k_proj_mat)
        torch.nn.init.normal_(m.v_proj_mat)
    inv = 1.0 / (10000.0 ** (np.arange(d // 2) / (d // 2)))
    freqs = torch.from_numpy(np.exp(1j * np.outer(np.arange(256.0), inv))[:, : wa.hkv.temporal_complex_dims(d)])
    hkv = wa.hkv.HKVCache(frame_seq_length=frame, page_size_frames=2, topk_pages=3, stage1_topk_chunks=2, hbm_max_chunks=hot, rerope=rerope)
    size, slots = window * frame, hsa[0].coarse_cache_size(window * frame)
    for c in range(2):
        cache = [{"k": make(size), "v": make(size), "k_coarse": make(slots), "v_coarse": make(slots),
                  "local_end_index": torch.tensor([size], device=dev()), "global_end_index": torch.tensor([size], device=dev())} for _ in range(layers)]
        # what lies behind an installed page must not reach its slots
        for block_cache in cache:
            block_cache["k"][:, 4 * frame] = float("nan")
        hkv.store(cache, prompt_embeds=make(1).float()[:, :, 0], current_start_frame=window * (c + 1), temporal_freqs=freqs)
    torch.cuda.synchronize()
    calls = []
    fused = wa.hkv.HKVCache._install_fused
    monkeypatch.setattr(wa.hkv.HKVCache, "_install_fused", lambda self, *a: calls.append(fused(self, *a)) or calls[-1])
    # pages of two frames and the last one of one; the last page of the second call does not fit and is left out
    for pairs, fits in ((((0, 1), (0, 3), (1, 0)), True), (((0, 0), (1, 1), (0, 3), (1, 0), (1, 3)), True)):
        start = [{n: t.clone() for n, t in b.items()} for b in cache]
        tokens = hkv.apply(cache, list(pairs), current_start_frame=40, temporal_freqs=freqs, hsa_modules=hsa)
        assert calls.pop() is fits and tokens % frame == 0
        with monkeypatch.context() as m:
            m.setattr(wa.hkv.HKVCache, "_install_fused", lambda self, *a: False)
            assert hkv.apply(start, list(pairs), current_start_frame=40, temporal_freqs=freqs, hsa_modules=hsa) == tokens
        for got, want in zip(cache, start):
            for name in want:
                assert torch.equal(got[name].view(torch.int16) if got[name].dtype == torch.bfloat16 else got[name],
                                   want[name].view(torch.int16) if want[name].dtype == torch.bfloat16 else want[name]), name


def test_pages_of_broken_frames_take_the_separate_kernels(monkeypatch):
    import worldattention_b200 as wa
    frame, heads, d = 16, 1, 128
    hkv = wa.hkv.HKVCache(frame_seq_length=frame, page_size_frames=2, hbm_max_chunks=1)
    hsa = [wa.hsa.HSAAttention(heads, d, block_size=64, proj_segment_len=frame).to(dev(), torch.bfloat16)]
    make = lambda n: torch.randn((1, n, heads, d), device=dev()).bfloat16()
    cache = [{"k": make(80), "v": make(80), "k_coarse": make(5), "v_coarse": make(5),
              "local_end_index": torch.tensor([80], device=dev()), "global_end_index": torch.tensor([80], device=dev())}]
    freqs = torch.polar(torch.ones(64, 22, dtype=torch.float64), torch.randn(64, 22, dtype=torch.float64))
    hkv.store(cache, prompt_embeds=make(1).float()[:, :, 0], current_start_frame=5, temporal_freqs=freqs)
    hkv.chunks[0]["page_spans"] = [(0, 32), (40, 72)]          # a page that does not start with a frame
    done = []
    fused = wa.hkv.HKVCache._install_fused
    monkeypatch.setattr(wa.hkv.HKVCache, "_install_fused", lambda self, *a: done.append(fused(self, *a)) or done[-1])
    assert hkv.apply(cache, [(0, 0), (0, 1)], current_start_frame=9, temporal_freqs=freqs, hsa_modules=hsa) == 64
    assert done == [False]


def _small_bank(frame=16, layers=2, frames=5):
    import worldattention_b200 as wa
    heads, d = 1, 128
    hkv = wa.hkv.HKVCache(frame_seq_length=frame, page_size_frames=2, hbm_max_chunks=1)
    hsa = [wa.hsa.HSAAttention(heads, d, block_size=64, proj_segment_len=frame).to(dev(), torch.bfloat16) for _ in range(layers)]
    size = frames * frame
    make = lambda n: torch.randn((1, n, heads, d), device=dev()).bfloat16()
    slots = hsa[0].coarse_cache_size(size)
    cache = [{"k": make(size), "v": make(size), "k_coarse": make(slots), "v_coarse": make(slots),
              "local_end_index": torch.tensor([size], device=dev()), "global_end_index": torch.tensor([size], device=dev())} for _ in range(layers)]
    freqs = torch.polar(torch.ones(64, 22, dtype=torch.float64), torch.randn(64, 22, dtype=torch.float64))
    hkv.store(cache, prompt_embeds=make(1).float()[:, :, 0], current_start_frame=frames, temporal_freqs=freqs)
    return hkv, hsa, cache, freqs


@pytest.mark.parametrize("start", [9, 9.0, 9.25, np.float32(9.25), torch.tensor(9), torch.tensor(9.25), "device"], ids=str)
@pytest.mark.parametrize("dtype", [torch.int64, torch.int32, torch.float32], ids=str)
def test_start_frame_of_any_number_type(start, dtype):
    hkv, hsa, cache, freqs = _small_bank()
    start = torch.tensor(9.25, device=dev()) if isinstance(start, str) else start
    for block in cache:
        block["global_end_index"] = block["global_end_index"].to(dtype)
    assert hkv.apply(cache, [(0, 1)], current_start_frame=start, temporal_freqs=freqs, hsa_modules=hsa) == 32
    for block in cache:
        assert torch.equal(block["global_end_index"].cpu(), torch.zeros(1, dtype=dtype).fill_(float(start) * 16))
        assert int(block["local_end_index"]) == 32


class _Compressor:
    """A module that offers what a compressed tier of its own kind needs, and nothing else."""

    def __init__(self, hsa):
        self.token_range_to_coarse, self.compress_kv_cache = hsa.token_range_to_coarse, hsa.compress_kv_cache


@pytest.mark.parametrize("tier", ["float32", "float32 in the last layer", "other strides of v", "channels apart"])
def test_a_tier_of_its_own_kind_asks_its_module_for_the_slots_only(tier):
    hkv, hsa, cache, freqs = _small_bank()
    modules = list(hsa)
    for m in hsa:
        torch.nn.init.normal_(m.k_proj_mat)
        torch.nn.init.normal_(m.v_proj_mat)
    for layer, block in enumerate(cache):
        if tier == "float32 in the last layer" and layer == 0:
            continue
        modules[layer] = _Compressor(hsa[layer])
        for name in ("k_coarse", "v_coarse") if tier != "other strides of v" else ("v_coarse",):
            if tier.startswith("float32"):
                block[name] = block[name].float()
            else:
                wide = torch.zeros(1, 5, 1, 256, device=dev(), dtype=torch.bfloat16)
                block[name] = wide[..., ::2] if tier == "channels apart" else wide[..., :128]
    assert hkv.apply(cache, [(0, 0), (0, 1)], current_start_frame=9, temporal_freqs=freqs, hsa_modules=modules) == 64
    for m, block in zip(hsa, cache):
        want = m.compress_kv_cache(block["k"][:, :64], block["v"][:, :64])
        for name, slots in zip(("k_coarse", "v_coarse"), want):
            assert torch.equal(block[name][:, :4], slots.to(block[name].dtype)) and not block[name][:, 4:].any()


def test_modules_may_be_keyed_by_layer():
    hkv, hsa, cache, freqs = _small_bank()
    assert hkv.apply(cache, [(0, 0)], current_start_frame=9, temporal_freqs=freqs, hsa_modules=dict(enumerate(hsa))) == 32


@pytest.mark.parametrize("view", ["conjugate", "imaginary part", "every other row", "band"])
def test_frequency_tables_on_the_device_in_every_view(view):
    """A table on the device is fetched without waiting; what comes of it is what the same values on the host give."""
    frame, heads, d = 16, 1, 128
    import worldattention_b200 as wa
    g = torch.Generator().manual_seed(3)
    base = torch.polar(torch.ones(4096, 64, dtype=torch.float64), torch.randn(4096, 64, generator=g, dtype=torch.float64))
    take = {"conjugate": lambda t: t[:, :22].conj(), "imaginary part": lambda t: t[:, :22].conj().imag, "every other row": lambda t: t[::2, :22],
            "band": lambda t: wa.hkv.temporal_band(t, d)}[view]
    k = torch.randn((1, 80, heads, d), generator=torch.Generator(device=dev()).manual_seed(4), device=dev()).bfloat16()
    indices = []
    for freqs in (take(base.to(dev())), take(base).resolve_conj().resolve_neg().clone()):
        hkv = wa.hkv.HKVCache(frame_seq_length=frame, page_size_frames=2, hbm_max_chunks=1)
        cache = [{"k": k.clone(), "v": k.clone(), "local_end_index": torch.tensor([80], device=dev()), "global_end_index": torch.tensor([80], device=dev())}]
        hkv.store(cache, prompt_embeds=torch.ones(1, 1, 8), current_start_frame=900, temporal_freqs=freqs)
        indices.append(hkv.chunks[0]["page_index"])
    assert torch.equal(*indices)


@pytest.mark.parametrize("frame", [16, 136])
@pytest.mark.parametrize("half_frames,pages,installed", [(14, 4, 7), (15, 3, 6), (14, 3, 6), (3, 1, None)])
def test_fused_install_at_the_end_of_the_cache(monkeypatch, frame, half_frames, pages, installed):
    """A page of two frames cut to one, a capacity that is no multiple of a frame, and one that cuts a frame (refused: its slots
    would be of a part of a segment)."""
    hkv, hsa, bank, freqs = _small_bank(frame, frames=8)
    capacity, slots = half_frames * frame // 2, (half_frames + 1) // 2 * hsa[0].proj_rank
    make = lambda n: torch.randn((1, n, 1, 128), device=dev()).bfloat16()
    for m in hsa:
        torch.nn.init.normal_(m.k_proj_mat)
        torch.nn.init.normal_(m.v_proj_mat)
    cache = [{"k": make(capacity), "v": make(capacity), "k_coarse": make(slots), "v_coarse": make(slots),
              "local_end_index": torch.tensor([0], device=dev()), "global_end_index": torch.tensor([0], device=dev())} for _ in hsa]
    other = [{n: t.clone() for n, t in b.items()} for b in cache]
    done = []
    fused = wa_cache()._install_fused
    monkeypatch.setattr(wa_cache(), "_install_fused", lambda self, *a: done.append(fused(self, *a)) or done[-1])
    call = lambda c: hkv.apply(c, [(0, p) for p in range(pages)], current_start_frame=9, temporal_freqs=freqs, hsa_modules=hsa)
    if installed is None:
        with pytest.raises(ValueError, match="segment-aligned"):
            call(cache)
        return
    assert call(cache) == installed * frame and done == [True]
    monkeypatch.setattr(wa_cache(), "_install_fused", lambda self, *a: False)
    assert call(other) == installed * frame
    for got, want in zip(cache, other):
        for name in want:
            assert torch.equal(got[name], want[name]), name
    for b, stored in zip(cache, hkv.tier.get(0)["v"]):
        assert torch.equal(b["v"][:, :installed * frame], stored[:, :installed * frame]) and not b["v"][:, installed * frame:].any()


def wa_cache():
    from worldattention_b200.hkv import HKVCache
    return HKVCache
