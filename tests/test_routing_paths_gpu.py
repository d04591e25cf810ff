"""The forward's routing against the stand-alone routing functions at the sizes where its kernels change: logits of 16-row and
128-key tiles and their remainders, and the best blocks of long rows picked in one or several pieces."""
import pytest
import torch

from tests.helpers import dev

pytestmark = pytest.mark.gpu
BLOCK, D = 8, 128


def _inputs(b, h, lq, lkv, seed, spread=1.0):
    g = torch.Generator(device=dev()).manual_seed(seed)
    draw = lambda n, s: (torch.randn(b, n, h, D, generator=g, device=dev()) * s).bfloat16()
    kc = draw(16, 1.0)
    proj = torch.zeros(1, 8, device=dev(), dtype=torch.bfloat16)      # not used: the compressed cache is given
    return (draw(lq, spread), draw(lkv, spread), draw(lkv, 1.0)), dict(k_coarse=kc, v_coarse=kc, k_proj_mat=proj, v_proj_mat=proj, block_size=BLOCK)


@pytest.mark.parametrize("b,h,nq,nkv", [(1, 16, 16, 256), (1, 32, 17, 129), (2, 4, 80, 127), (1, 3, 81, 300), (1, 1, 33, 2049),
                                        (1, 40, 1, 1700), (1, 2, 97, 513), (1, 1, 15, 4096), (1, 1, 2, 128),
                                        # on 148 SMs a CTA of the logits kernel holds one row tile of those above from 65 536 logits
                                        # on, and two, three, four and five of these
                                        (1, 40, 17, 129), (1, 24, 97, 129), (1, 40, 49, 300), (1, 40, 65, 300),
                                        # a key per thread, and passes through shared memory beyond
                                        (1, 3, 5, 257), (1, 3, 70, 512), (1, 3, 5, 513), (1, 3, 70, 1024),
                                        # short rows: a CTA per head, one, two or four keys per lane, and just beyond
                                        (1, 3, 1, 1), (2, 3, 7, 19), (1, 2, 37, 37), (1, 2, 64, 128), (2, 2, 32, 64), (1, 1, 16, 8), (1, 2, 33, 33),
                                        (4, 2, 16, 127), (4, 2, 8, 127), (1, 2, 32, 128), (1, 2, 33, 80), (1, 2, 64, 64),
                                        (1, 2, 65, 40), (1, 2, 64, 129),
                                        # ... spread over clusters of one, two, four and eight
                                        (1, 2, 8, 19), (1, 3, 9, 65), (1, 2, 17, 128), (1, 3, 57, 33)])
@pytest.mark.parametrize("ragged", [0, 3])
def test_forward_routing_equals_the_separate_functions(b, h, nq, nkv, ragged):
    from worldattention_b200.hsa import routing as R
    from worldattention_b200.hsa import hsa_attention
    lq, lkv = nq * BLOCK - ragged, nkv * BLOCK - ragged
    qkv, kwargs = _inputs(b, h, lq, lkv, nq + nkv)
    _, (index, num, thresholds, _) = hsa_attention(*qkv, return_routing=True, **kwargs)
    pooled = [R.block_mean_pool(R.pad_to_len(t, n * BLOCK).transpose(1, 2).contiguous(), length, n, BLOCK).float()
              for t, n, length in ((qkv[0], nq, lq), (qkv[1], nkv, lkv))]
    want = R.build_block_routing(R.block_attention_map(*pooled), 0.35, 1.0)
    assert torch.equal(index, want.index) and torch.equal(num, want.num) and torch.equal(thresholds, want.thresholds)


@pytest.mark.parametrize("topk", [(4500, 2049), (2048, 1), (1025, 512), (5000, 0), (4097, 33)])
@pytest.mark.parametrize("spread", [1.0, 0.0])      # 0: every probability is the same, the order is the ids'
def test_best_blocks_of_long_rows(topk, spread):
    from worldattention_b200.hsa import hsa_attention
    qkv, kwargs = _inputs(1, 2, 3 * BLOCK, 5000 * BLOCK, 5, spread)
    counts = torch.tensor(topk, dtype=torch.int32)
    picked = hsa_attention(*qkv, topk_per_head=counts, **kwargs)
    whole, (_, num, _, _) = hsa_attention(*qkv, topk_per_head=counts, return_routing=True, **kwargs)
    assert num.unique().tolist() == sorted(set(topk)) and torch.equal(picked, whole)


# fixed counts: one row per CTA of 128 (logits ready), 256 or 512 threads, up to 32 blocks per thread; few and many best blocks
# collected, ordered by counting, by sorting, or (beyond 2048) in pieces
@pytest.mark.parametrize("nq,nkv,topk", [(3, 1, (1, 0, 1)), (3, 129, (4, 129, 0)), (90, 256, (16, 127, 256)), (90, 255, (1, 33, 128)),
                                         (60, 511, (32, 129, 511)), (3, 257, (31, 256, 257)), (30, 2048, (8, 257, 2047)),
                                         (37, 37, (4, 37, 1)), (64, 128, (31, 33, 128)), (2, 2049, (64, 513, 2049)), (2, 4097, (32, 512, 3000)), (2, 8193, (1, 100, 600)),
                                         (2, 16384, (32, 16384, 2048))])
@pytest.mark.parametrize("spread", [1.0, 0.0])
def test_best_blocks_by_count(nq, nkv, topk, spread):
    from worldattention_b200.hsa import hsa_attention
    qkv, kwargs = _inputs(1, 3, nq * BLOCK, nkv * BLOCK - 3, nkv, spread)
    counts = torch.tensor(topk, dtype=torch.int32)
    picked = hsa_attention(*qkv, topk_per_head=counts, **kwargs)
    whole, (_, num, _, _) = hsa_attention(*qkv, topk_per_head=counts, return_routing=True, **kwargs)
    assert num.unique().tolist() == sorted(set(topk)) and torch.equal(picked, whole)


# beside the compression of the call's own keys and values (projections of zeros: the coarse blocks are exact zeros): short rows by
# one or two CTAs per head; pairs of 64-token blocks, which the routing then orders by counts, in every routing kernel
@pytest.mark.parametrize("b,h,nq,nkv,block", [(1, 3, 1, 1, 8), (1, 3, 8, 33, 8), (1, 3, 9, 64, 8), (1, 3, 17, 65, 8), (1, 3, 64, 128, 8), (2, 3, 3, 22, 8),
                                              (2, 3, 32, 64, 8), (1, 40, 9, 5, 64), (2, 20, 4, 7, 64), (1, 3, 101, 30, 64), (1, 2, 75, 129, 64)])
@pytest.mark.parametrize("fixed", [False, True])
def test_routing_beside_the_compression(b, h, nq, nkv, block, fixed):
    from worldattention_b200.hsa import hsa_attention
    qkv, kwargs = _inputs(b, h, nq * block - 1, nkv * block, nkv)
    proj = torch.zeros(1, nkv * block, device=dev(), dtype=torch.bfloat16)
    kwargs.update(block_size=block, k_proj_mat=proj, v_proj_mat=proj, k_coarse=qkv[1].new_zeros(b, 16, h, D), v_coarse=qkv[1].new_zeros(b, 16, h, D))
    if fixed:
        kwargs.update(topk_per_head=torch.tensor([1, nkv, nkv // 2], dtype=torch.int32).repeat(h)[:h])
    given = hsa_attention(*qkv, **kwargs)
    kwargs.update(k_coarse=None, v_coarse=None)
    assert torch.equal(hsa_attention(*qkv, **kwargs), given)


# the same with float32 projections, which a kernel of fewer CTAs multiplies: its shares per segment (of 64 tokens and more) are cut to
# fit beside the routing's CTAs, which keep their SMs to themselves where all fit; 16 rows and 48 keys are the most of one routing CTA
@pytest.mark.parametrize("b,h,q_len,segments,seg,block", [(1, 8, 600, 3, 635, 64), (1, 12, 1000, 4, 760, 64), (1, 12, 1024, 4, 768, 64), (1, 12, 1025, 4, 769, 64),
                                                          (1, 24, 700, 3, 300, 64), (1, 16, 128, 2, 100, 128), (1, 3, 513, 5, 640, 64), (2, 12, 200, 2, 130, 64),
                                                          (1, 24, 1100, 12, 70, 64), (1, 74, 64, 1, 600, 64),
                                                          # ... and one of 32 warps beside which more of the compression fits
                                                          (1, 16, 1071, 2, 1071, 64), (1, 16, 1100, 1, 1100, 64)])
@pytest.mark.parametrize("zeros", [True, False])
def test_compression_that_fits_beside_the_routing(b, h, q_len, segments, seg, block, zeros):
    from tests.helpers import attention_error, to_np
    from worldattention_b200.hsa import HSAAttention
    g = torch.Generator(device=dev()).manual_seed(seg)
    draw = lambda n: torch.randn(b, n, h, D, generator=g, device=dev()).bfloat16()
    q, k, v = draw(q_len), draw(segments * seg - 3), draw(segments * seg - 3)
    hsa = HSAAttention(h, D, block_size=block, proj_segment_len=seg).to(dev())
    with torch.no_grad():
        for p in (hsa.k_proj_mat, hsa.v_proj_mat):
            p.copy_(torch.randn(p.shape, generator=g, device=dev()) * (0 if zeros else 0.1))
        kc, vc = hsa.compress_kv_cache(k, v)
        out, given = hsa(q, k, v), hsa(q, k, v, k_coarse=kc, v_coarse=vc)
    if zeros:
        assert torch.equal(out, given)
    else:       # float32 sums of another order: a slot may round to the bf16 number next to it
        max_abs, mean_rel = attention_error(to_np(out), to_np(given))
        assert max_abs < 2e-2 and mean_rel < 1e-3
