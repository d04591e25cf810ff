"""Page scores and top-k at the sizes where the kernel changes: pages per warp, a key per thread, bitonic passes, longer banks, odd rows."""
import pytest
import torch

from tests.helpers import dev

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("pages,groups,dim,topk", [(1, 1, 1536, 1), (14, 1, 1536, 4), (15, 3, 128, 15), (65, 12, 128, 16), (512, 2, 132, 512),
                                                   (513, 2, 4, 20), (4096, 1, 128, 64), (4097, 1, 128, 33), (700, 2, 130, 9), (40, 1, 4100, 3)])
def test_scores_and_order(pages, groups, dim, topk):
    from worldattention_b200.hkv.retrieval import score_and_topk, score_and_topk_layers
    g = torch.Generator(device=dev()).manual_seed(pages)
    index = torch.randn((2, pages, groups * dim), generator=g, device=dev())
    index[:, pages // 2] = index[:, 0]                       # equal scores: the lower id first
    query = torch.randn((2, groups * dim), generator=g, device=dev())
    scores, ids, vals = score_and_topk_layers(query, index, topk, groups=groups)
    want = (index.double().view(2, pages, groups, dim) * query.double().view(2, 1, groups, dim)).sum(-1).transpose(1, 2).float() / dim ** 0.5
    # float64 sums: another order moves a score across a float32 rounding at most
    torch.testing.assert_close(scores, want, rtol=2 ** -22, atol=1e-12)
    order = torch.sort(scores, dim=-1, descending=True, stable=True)[1][..., :topk]
    assert torch.equal(ids.long(), order) and torch.equal(vals, scores.gather(-1, order))
    one = score_and_topk(query[1], index[1], topk, groups=groups)
    assert torch.equal(one[0], scores[1]) and torch.equal(one[1], ids[1]) and torch.equal(one[2], vals[1])
