"""Block means of inputs above half a gigabyte, which the TMA stream reads with one consumer group more."""
import pytest
import torch

from tests.helpers import dev

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("length,block", [(2800 * 64 + 40, 64), (1450 * 128, 128)])
def test_long_inputs(length, block):
    from worldattention_b200.hsa.routing import block_mean_pool
    heads, d, n = 12, 128, -(-length // block)
    assert length * heads * d * 2 > 512 << 20
    g = torch.Generator(device=dev()).manual_seed(block)
    x = torch.zeros(1, n * block, heads, d, device=dev(), dtype=torch.bfloat16)
    x[:, :length] = torch.randn((1, length, 1, d), generator=g, device=dev()).bfloat16() * torch.arange(1, heads + 1, device=dev())[:, None]
    got = block_mean_pool(x.transpose(1, 2), length, n, block).float()
    for first in range(0, n, 256):                       # float64 sums, exact for these values
        sums = x.view(n, block, heads, d)[first: first + 256].double().sum(1)
        if length % block == 0:
            want = (sums / block).float().bfloat16().float()
        else:
            real = torch.tensor([min(block, length - i * block) for i in range(first, min(n, first + 256))], device=dev(), dtype=torch.float32)
            want = sums.float().bfloat16().float() / real[:, None, None]
        assert torch.equal(got[0, :, first: first + 256].transpose(0, 1), want)
