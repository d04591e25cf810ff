"""Float32 layers with as many rows as the chip has SMs round their keys once for all of them; rows are taken heaviest first and the
linear branch runs beside the sparse one in every float32 layer that routes for itself.  Heads are independent, so a call with fewer heads,
whose blocks round the keys they select themselves, must give the same bits; so must the branches launched one by one, which know neither
the rounding nor the order nor the overlap."""
import pytest
import torch

from tests.helpers import dev

pytestmark = pytest.mark.gpu
D = 128


@pytest.mark.parametrize("batch,q_len,kv_len,block", [(1, 16 * 64, 40 * 64, 64), (2, 7 * 64 - 5, 19 * 64 - 3, 64), (1, 14 * 128 - 1, 900, 128)])
@pytest.mark.parametrize("coarse", [False, True])
@pytest.mark.parametrize("wide", [False, True])        # keys that are a slice of a cache with a longer row
def test_rounding_keys_once_changes_nothing(batch, q_len, kv_len, block, coarse, wide):
    from worldattention_b200.hsa import hsa_attention
    heads, part = 12, 3
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    rows = batch * -(-q_len // block)
    assert heads * rows >= sms > part * rows
    g = torch.Generator(device=dev()).manual_seed(q_len)
    draw = lambda n, h=heads: torch.randn(batch, n, h, D, generator=g, device=dev())
    q, k, v = draw(q_len), draw(kv_len, heads + wide)[:, :, :heads], draw(kv_len, heads + wide)[:, :, :heads]
    seg = 320
    proj = torch.randn(-(-seg // block), seg, generator=g, device=dev()) * 0.05
    lin = torch.nn.Linear(D, D).to(dev())
    kwargs = dict(k_proj_mat=proj, v_proj_mat=proj, gate_lin=lin, block_size=block, proj_segment_len=seg)
    kc, vc = (draw(50), draw(50)) if coarse else (None, None)
    cut = lambda t: None if t is None else t[:, :, :part]
    with torch.no_grad():
        whole = hsa_attention(q, k, v, k_coarse=kc, v_coarse=vc, **kwargs)
        few = hsa_attention(cut(q), cut(k), cut(v), k_coarse=cut(kc), v_coarse=cut(vc), **kwargs)
    if coarse:
        assert torch.equal(whole[:, :, :part], few)
    else:       # the compression splits a segment over more CTAs where a call has fewer heads: float32 sums in another order
        assert float((whole[:, :, :part] - few).abs().max()) < 1e-5


@pytest.mark.parametrize("q_len,kv_len,block", [(16 * 64, 40 * 64, 64), (7 * 64 - 5, 19 * 64 - 3, 64), (14 * 128 - 1, 900, 128), (200, 1170, 64)])
@pytest.mark.parametrize("fixed", [False, True])
def test_one_call_equals_its_branches_one_by_one(q_len, kv_len, block, fixed):
    from worldattention_b200.hsa import hsa_attention
    from worldattention_b200.hsa.branches import gate_combine, linear_branch, sparse_branch
    heads = 12
    g = torch.Generator(device=dev()).manual_seed(q_len + fixed)
    draw = lambda n: torch.randn(1, n, heads, D, generator=g, device=dev())
    q, k, v, kc, vc = draw(q_len), draw(kv_len), draw(kv_len), draw(50), draw(50)
    lin = torch.nn.Linear(D, D).to(dev())
    counts = torch.randint(1, 9, (heads,), generator=g, device=dev()).int() if fixed else None
    kwargs = dict(k_coarse=kc, v_coarse=vc, k_proj_mat=None, v_proj_mat=None, gate_lin=lin, block_size=block, topk_per_head=counts)
    with torch.no_grad():
        plain = hsa_attention(q, k, v, **kwargs)
        out, (index, num, _, _) = hsa_attention(q, k, v, return_routing=True, **kwargs)
        sparse = sparse_branch(q, k, v, index, num, block, lse=False, round_output_bf16=True)[0]
        want = gate_combine(q, sparse, linear_branch(q, kc, vc, lse=False)[0], lin, round_bf16=False)
    assert torch.equal(plain, out) and torch.equal(out, want)
