"""64-token routing blocks with two query blocks per work item (more blocks than SMs) against the oracle and the library's
float32 path: odd numbers of query blocks, a ragged last block, pairs with unequal, equal, disjoint and empty selections."""
import math

import numpy as np
import pytest
import torch

from oracle import hsa_oracle as O
from tests.helpers import attention_error, dev, to_gpu, to_np

pytestmark = pytest.mark.gpu
D, BLOCK = 128, 64
MAX_ABS, MEAN_REL = 2e-2, 1e-2      # as for the other block sizes (bf16 operands and result)


def _inputs(seed, bsz, heads, q_len, kv_len, scale):
    rng = np.random.default_rng(seed)
    draw = lambda n, s: O.bf16_round((rng.standard_normal((bsz, n, heads, D)) * s).astype(np.float32))
    return rng, draw(q_len, scale), draw(kv_len, scale), draw(kv_len, 1.0)


def _close(got, want, v):
    # Both branches are averages of v.  The sparse one and the result are each rounded to bf16, and a value next to a rounding
    # boundary may go either way: one step of the largest |v| for each of the two, where that is more than the usual bound.
    step = 2.0 ** (math.floor(math.log2(np.abs(v).max())) - 7)
    max_abs, mean_rel = attention_error(got, want)
    assert max_abs <= max(MAX_ABS, 2 * step) and mean_rel < MEAN_REL


@pytest.mark.parametrize("bsz,heads,q_len,kv_len,seg,topk,scale", [
    (1, 12, 13 * BLOCK, 1000, 250, [3, 1, 16, 5, 2, 7, 9, 4, 6, 8, 11, 2], 0.3),   # 13 blocks a head: the last item is half empty
    (1, 30, 5 * BLOCK + 7, 700, 350, [0, 1, 2] * 10, 0.3),                         # ragged last block, empty selections
    (2, 16, 6 * BLOCK, 2048, 512, None, 0.6),                                      # counts from the mass: unequal within a pair
    (1, 40, 4 * BLOCK - 1, 4096, 1024, [64] * 40, 3.0),                            # large logits: running maxima are outgrown
])
def test_paired_query_blocks(bsz, heads, q_len, kv_len, seg, topk, scale):
    import worldattention_b200 as wa
    assert bsz * heads * math.ceil(q_len / BLOCK) > torch.cuda.get_device_properties(0).multi_processor_count
    rng, q, k, v = _inputs(heads, bsz, heads, q_len, kv_len, scale)
    if topk is None:       # blocks that differ from one another, so that rows of a head keep different shares of them
        q, k = (O.bf16_round(x + np.repeat(rng.standard_normal((bsz, x.shape[1] // BLOCK, heads, D)).astype(np.float32), BLOCK, axis=1)) for x in (q, k))
    rank = math.ceil(seg / BLOCK)
    e = O.bf16_round((rng.standard_normal((rank, seg)) * 0.05).astype(np.float32))
    gw, gb = O.bf16_round((rng.standard_normal((D, D)) * 0.05).astype(np.float32)), (rng.standard_normal((D,)) * 0.3).astype(np.float32)
    lin = torch.nn.Linear(D, D).to(dev())
    with torch.no_grad():
        lin.weight.copy_(to_gpu(gw)); lin.bias.copy_(to_gpu(gb))
    kwargs = dict(k_proj_mat=to_gpu(e, "bf16"), v_proj_mat=to_gpu(e, "bf16"), gate_lin=lin, block_size=BLOCK, proj_segment_len=seg,
                  topk_per_head=None if topk is None else torch.tensor(topk, dtype=torch.int32), return_routing=True)
    args = [to_gpu(x, "bf16") for x in (q, k, v)]
    out, (index, num, thr, used) = wa.hsa.hsa_attention(*args, check_status=True, **kwargs)
    assert used
    ref, (index_g, num_g, thr_g, used_g) = wa.hsa.hsa_attention(*args, force_generic=True, **kwargs)
    assert not used_g and torch.equal(index, index_g) and torch.equal(num, num_g)
    if topk is None:
        n = num.reshape(bsz, heads, -1)
        assert bool((n[..., 0:-1:2] != n[..., 1::2]).any()), "the inputs should give a pair unequal counts"
    _close(to_np(out), to_np(ref), v)
    want = O.hsa_attention(q, k, v, k_proj_mat=e, v_proj_mat=e, gate_weight=gw, gate_bias=gb, block_size=BLOCK, proj_segment_len=seg,
                           dtype="bf16", topk_per_head=topk)
    _close(to_np(out), want, v)
    # no state is carried from one launch to the next
    again, _ = wa.hsa.hsa_attention(*args, **kwargs)
    assert torch.equal(out, again)


def test_a_block_that_only_the_neighbour_selects_does_not_reach_a_query_block():
    # one selected block per query block: an infinity in a key block's values reaches exactly the query blocks that chose it
    import worldattention_b200 as wa
    heads, q_len, kv_len = 20, 10 * BLOCK, 12 * BLOCK
    rng, q, k, v = _inputs(5, 1, heads, q_len, kv_len, 0.4)
    v[0, 3 * BLOCK + 5, :, 17] = np.inf
    kc, vc = (to_gpu(O.bf16_round(rng.standard_normal((1, 24, heads, D)).astype(np.float32)), "bf16") for _ in range(2))
    out, (index, num, _, used) = wa.hsa.hsa_attention(
        *[to_gpu(x, "bf16") for x in (q, k, v)], k_coarse=kc, v_coarse=vc, k_proj_mat=None, v_proj_mat=None, gate_lin=None, block_size=BLOCK,
        topk_per_head=torch.ones(heads, dtype=torch.int32), return_routing=True)
    assert used
    chose = index[0, :, :, 0] == 3                                                # [heads, query blocks]
    hit = ~torch.isfinite(out[0, :, :, 17]).reshape(-1, BLOCK, heads)              # [query blocks, rows, heads]
    assert chose.any() and not chose.all()
    assert torch.equal(hit.any(dim=1).T, chose)
    assert bool(torch.isfinite(out[..., :17]).all()) and bool(torch.isfinite(out[..., 18:]).all())


def test_partial_results_of_pairs_with_supplied_routing():
    # the two branches separately, with a routing of the caller's own: overlapping, disjoint, empty and repeated selections
    from worldattention_b200.hsa.branches import hsa_partials
    heads, q_len, kv_len = 24, 8 * BLOCK - 9, 40 * BLOCK - 17
    rng, q, k, v = _inputs(11, 1, heads, q_len, kv_len, 0.4)
    kc, vc = (to_gpu(O.bf16_round(rng.standard_normal((1, 130, heads, D)).astype(np.float32)), "bf16") for _ in range(2))
    args = [to_gpu(x, "bf16") for x in (q, k, v)]
    index = torch.stack([torch.randperm(40) for _ in range(heads * 8)]).view(1, heads, 8, 40).int()
    num = torch.randint(0, 41, (1, heads, 8)).int()
    index[0, 0, 1] = index[0, 0, 0]                       # the same list for both
    num[0, 0, :2] = 17
    index[0, 1, 0, :20], index[0, 1, 1, :20] = torch.arange(20), torch.arange(20, 40)      # nothing in common
    num[0, 1, :2] = 20
    index[0, 2, 0, :4] = torch.tensor([3, 3, 5, 3])       # a block named more than once counts that often
    index[0, 2, 1, :4] = torch.tensor([5, 3, 5, 7])
    num[0, 2, :2] = 4
    got = hsa_partials(*args, kc, vc, index.to(dev()), num.to(dev()), BLOCK)
    want = hsa_partials(*args, kc, vc, index.to(dev()), num.to(dev()), BLOCK, force_generic=True)
    assert got[4] and not want[4]
    for a, b in zip(got[:4], want[:4]):
        a, b = to_np(a), to_np(b)
        assert np.array_equal(np.isinf(a), np.isinf(b))
        a, b = np.where(np.isinf(a), 0, a), np.where(np.isinf(b), 0, b)
        assert attention_error(a, b)[0] < MAX_ABS and attention_error(a, b)[1] < MEAN_REL
