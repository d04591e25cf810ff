"""The native host module's own work: what it refuses, how it reads its arguments, and the workspaces it keeps."""
import pytest
import torch

from tests.helpers import dev

pytestmark = pytest.mark.gpu
D = 128


def _inputs(lq=130, lkv=200, heads=2, block=64, seed=0):
    g = torch.Generator(device=dev()).manual_seed(seed)
    make = lambda n: torch.randn((1, n, heads, D), generator=g, device=dev()).to(torch.bfloat16)
    proj = torch.full((-(-lkv // block), lkv), 1 / block, device=dev(), dtype=torch.bfloat16)
    return dict(q=make(lq), k=make(lkv), v=make(lkv), k_proj_mat=proj, v_proj_mat=proj, proj_segment_len=lkv, block_size=block)


def _attend(q, k, v, **options):
    from worldattention_b200.hsa import hsa_attention
    with torch.no_grad():
        return hsa_attention(q, k, v, **options)


@pytest.mark.parametrize("routing", [False, True])
@pytest.mark.parametrize("block", [0, -1, 1 << 32])
def test_block_sizes_that_are_none(block, routing):
    with pytest.raises(ValueError):
        _attend(**{**_inputs(), "block_size": block}, return_routing=routing)
