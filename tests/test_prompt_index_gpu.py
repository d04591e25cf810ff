"""The prompt index in two launches against float64, and the tensor expressions it leaves other layouts to."""
import pytest
import torch

from tests.helpers import dev

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("b,tokens,dim", [(1, 512, 4096), (1, 1, 8), (2, 31, 72), (3, 257, 1528), (1, 300, 12)])
def test_prompt_index(dtype, b, tokens, dim):
    from worldattention_b200.hkv.retrieval import prompt_index
    g = torch.Generator(device=dev()).manual_seed(dim)
    x = torch.randn((b, tokens + 2, dim), generator=g, device=dev()).to(dtype)
    for t in (x[:, :tokens], x[:, 2:], x.transpose(1, 2).contiguous().transpose(1, 2)[:, :tokens]):
        mean = t.double().mean(1).mean(0)
        # the means are rounded to float32 (2^-24 of the largest value of a column's terms), the quotient once more
        assert float((prompt_index(t).double() - mean / mean.norm()).abs().max()) < 2e-6
    zero = prompt_index(torch.zeros(1, 4, 16, device=dev(), dtype=dtype))
    assert not zero.any() and bool(prompt_index(torch.full((1, 4, 16), float("nan"), device=dev(), dtype=dtype)).isnan().all())


def test_prompt_index_under_function_transforms():
    from worldattention_b200.hkv.retrieval import prompt_index
    x = torch.randn((3, 2, 16, 8), generator=torch.Generator(device=dev()).manual_seed(1), device=dev())
    batched = torch.vmap(prompt_index)(x)
    torch.testing.assert_close(batched, torch.stack([prompt_index(t) for t in x]), rtol=0, atol=2e-6)
    mean = lambda t: t.mean(1).mean(0)
    want = torch.func.jvp(lambda t: mean(t) / mean(t).norm(), (x[0].double(),), (x[1].double(),))
    for got in (torch.func.jvp(prompt_index, (x[0],), (x[1],)), _dual(prompt_index, x[0], x[1])):
        for a, b in zip(got, want):      # float32 sums of 16 values near 1 and a quotient
            torch.testing.assert_close(a.double(), b, rtol=0, atol=2e-6)


def _dual(f, x, tangent):
    from torch.autograd import forward_ad
    with forward_ad.dual_level():
        return tuple(forward_ad.unpack_dual(f(forward_ad.make_dual(x, tangent))))


def test_prompt_index_is_recorded_as_tensor_expressions():
    from torch.fx.experimental.proxy_tensor import make_fx
    from torch.utils.flop_counter import FlopCounterMode
    from worldattention_b200.hkv.retrieval import prompt_index
    first, other = (torch.randn((2, 16, 8), generator=torch.Generator(device=dev()).manual_seed(s), device=dev()) for s in (1, 2))
    recorded = [torch.jit.trace(prompt_index, first), make_fx(prompt_index)(first), torch.compile(prompt_index, backend="eager", fullgraph=True)]
    for f in recorded:       # of another input: a result that was computed while recording would be the first one's
        torch.testing.assert_close(f(other), prompt_index(other), rtol=0, atol=2e-6)
    with FlopCounterMode(display=False):
        torch.testing.assert_close(prompt_index(first), recorded[1](first), rtol=0, atol=2e-6)
