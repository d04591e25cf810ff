"""HKV kernels at the sizes where their work is split: page centroids over clusters, stored windows, tail clearing and whole-chunk
installs in one launch each."""
import numpy as np
import pytest
import torch

from oracle import hkv_oracle as K
from tests.helpers import dev, to_gpu, to_np

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bsz,heads,tokens,page,frame", [(1, 12, 700, 300, 100), (2, 3, 37, 16, 5), (1, 2, 9, 9, 3), (1, 4, 5000, 10, 10)])
def test_page_centroids(bsz, heads, tokens, page, frame):
    # few long pages (split over a cluster), pages shorter than a cluster's shares, one page, and more pages than CTAs per chip
    import worldattention_b200 as wa
    rng = np.random.default_rng(tokens)
    keys = rng.standard_normal((bsz, tokens, heads, 128)).astype(np.float32)
    keys = to_np(to_gpu(keys, "bf16"))
    spans = [(s, min(s + page, tokens)) for s in range(0, tokens, page)]
    inv = 1.0 / (10000.0 ** (np.arange(64) / 64))
    freqs = np.exp(1j * np.outer(np.arange(1024.0), inv))[:, : wa.hkv.temporal_complex_dims(128)]
    got = wa.hkv.page_key_index(to_gpu(keys, "bf16"), spans, frame_seq_length=frame, start_frame=2, temporal_freqs=torch.from_numpy(freqs))
    want = K.page_key_index(keys, spans, frame_seq_length=frame, start_frame=2, temporal_freqs=freqs, dtype="bf16")
    # float64 sums: the order of the additions can move a mean across a float32 rounding at most
    np.testing.assert_allclose(to_np(got), want, rtol=2 ** -23, atol=1e-9)


@pytest.mark.parametrize("hot,dtype,coarse_dtype", [(2, torch.bfloat16, torch.bfloat16), (0, torch.bfloat16, torch.bfloat16),
                                                    (1, torch.float32, torch.float32), (1, torch.bfloat16, torch.float32)])
def test_apply_installs_pages_and_clears_the_rest(hot, dtype, coarse_dtype):
    # two chunks of which `hot` lie in HBM (the others on the host), batch of two, layers in separate allocations
    import worldattention_b200 as wa
    frame, heads, d, cap, layers = 20, 2, 64, 200, 3
    g = torch.Generator(device=dev()).manual_seed(1)
    hsa = [wa.hsa.HSAAttention(heads, d, block_size=64, proj_segment_len=frame).to(dev(), dtype) for _ in range(layers)]
    for m in hsa:
        torch.nn.init.normal_(m.k_proj_mat)
        torch.nn.init.normal_(m.v_proj_mat)
    inv = 1.0 / (10000.0 ** (np.arange(32) / 32))
    freqs = torch.from_numpy(np.exp(1j * np.outer(np.arange(256.0), inv))[:, : wa.hkv.temporal_complex_dims(d)])
    hkv = wa.hkv.HKVCache(frame_seq_length=frame, page_size_frames=2, topk_pages=3, stage1_topk_chunks=2, hbm_max_chunks=hot, rerope=False)
    make = lambda n, t: torch.randn((2, n, heads, d), generator=g, device=dev()).to(t)
    slots = hsa[0].coarse_cache_size(cap)
    stored = []
    for c in range(2):
        cache = [{"k": make(cap, dtype), "v": make(cap, dtype), "k_coarse": make(slots, coarse_dtype), "v_coarse": make(slots, coarse_dtype),
                  "local_end_index": torch.tensor([cap - 20 * c], device=dev()), "global_end_index": torch.tensor([cap], device=dev())} for _ in range(layers)]
        chunk = hkv.store(cache, prompt_embeds=make(1, torch.float32)[:, :, 0], current_start_frame=10 * (c + 1), temporal_freqs=freqs)
        stored.append([{n: b[n].clone() for n in ("k", "v")} for b in cache])
        torch.cuda.synchronize()
        for layer in range(layers):          # a chunk holds the populated rows of every layer
            for name in ("k", "v"):
                assert torch.equal(hkv.tier.get(chunk)[name][layer].to(dev()), cache[layer][name][:, : cap - 20 * c])
    pairs = [(0, 1), (0, 4), (1, 0)]
    tokens = hkv.apply(cache, pairs, current_start_frame=40, temporal_freqs=freqs, hsa_modules=hsa)
    assert tokens == 3 * 2 * frame
    filled = hsa[0].token_range_to_coarse(0, tokens)[1]
    for layer, block in enumerate(cache):
        for name in ("k", "v"):
            want = torch.zeros_like(block[name])
            for i, (c, page) in enumerate(pairs):
                want[:, 40 * i: 40 * (i + 1)] = stored[c][layer][name][:, 40 * page: 40 * (page + 1)]
            assert torch.equal(block[name], want)
            assert not block[name + "_coarse"][:, filled:].any() and bool(block[name + "_coarse"][:, :filled].any())
        kc, vc = hsa[layer].compress_kv_cache(block["k"][:, :tokens], block["v"][:, :tokens])
        assert torch.equal(block["k_coarse"][:, :filled], kc.to(coarse_dtype)) and torch.equal(block["v_coarse"][:, :filled], vc.to(coarse_dtype))
        assert int(block["local_end_index"]) == tokens and int(block["global_end_index"]) == 40 * frame


@pytest.mark.parametrize("dtype,row,pad,first,counts", [(torch.bfloat16, 1536, 0, 0, (40, 1, 0, 700)), (torch.bfloat16, 6, 2, 1, (5, 3000)),
                                                        (torch.bfloat16, 16, 8, 3, (9,)), (torch.float32, 8, 0, 0, (300, 2)),
                                                        (torch.float32, 6, 1, 1, (2000, 7)), (torch.float32, 4, 0, 0, (1,) * 65537)])
def test_clear_rows_clears_its_rows_and_nothing_else(dtype, row, pad, first, counts):
    # 16-byte pieces, rows and addresses that are not multiples of them, gaps between rows, records without rows, more than a launch takes
    from worldattention_b200.hkv.install import RECORD_DTYPE, clear_rows_device
    stride, size = row + pad, torch.empty((), dtype=dtype).element_size()
    starts = np.cumsum([0] + [n + 2 for n in counts])            # two rows of others between the records
    x = torch.full((first + int(starts[-1]) * stride,), 3.0, dtype=dtype, device=dev())
    records = np.zeros(len(counts), dtype=RECORD_DTYPE)
    records["dst"] = [x.data_ptr() + (first + int(s) * stride) * size for s in starts[:-1]]
    records["dst_stride"], records["n_tokens"], records["src"] = stride, counts, 0
    clear_rows_device(torch.from_numpy(records.view(np.uint8)).to(dev()), max_tokens=max(counts), row_elems=row, elem_size=size)
    want = torch.full((int(starts[-1]), stride), 3.0)
    for s, n in zip(starts, counts):
        want[int(s): int(s) + n, :row] = 0
    assert bool((x[:first] == 3.0).all()) and torch.equal(x[first:].view(-1, stride).float().cpu(), want)


@pytest.mark.parametrize("heads,pages,page", [(12, 14, 50), (12, 21, 33), (12, 30, 7), (1, 460, 384), (1, 2100, 40)])
def test_page_centroids_by_four_three_two_and_one(heads, pages, page):
    # CTAs per page: four, three and two resident ones, two over several waves, one
    test_page_centroids(1, heads, pages * page - page // 3, page, 11)
