"""Float32 layers with as many rows as the chip has SMs: keys rounded once for all of them, rows heaviest first, the linear branch
beside the sparse one.  Heads are independent, so a call with fewer heads, which does none of this, must give the same bits."""
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
