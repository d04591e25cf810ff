"""The feed-forward of a block: an `nn.Sequential` like any other, and its GELU inside the first product where nothing can tell."""
import pytest
import torch
import torch.nn as nn
import torch.nn.functional as F

from tests.helpers import dev


def _ffn(dim=256, hidden=512):
    from worldattention_b200.causal_dit import CausalDiT, DiTConfig
    torch.manual_seed(0)
    return CausalDiT(DiTConfig(dim=dim, heads=dim // 128, ffn_dim=hidden, layers=1, text_dim=64)).blocks[0].ffn


def test_it_can_be_sliced_and_extended():
    ffn, x = _ffn(), torch.randn(1, 3, 256)
    assert ffn[:2](x).shape == (1, 3, 512)
    want = ffn(x)
    assert torch.equal(ffn.append(nn.Dropout(0.0))(x), want)


@pytest.mark.gpu
@pytest.mark.parametrize("tokens,dim,hidden", [(1, 256, 512), (33, 256, 520), (777, 1536, 8960), (4680, 1536, 8960)])
def test_distance_from_float64_is_no_larger(tokens, dim, hidden):
    from worldattention_b200.causal_dit import feed_forward
    ffn = _ffn(dim, hidden).to(dev(), torch.bfloat16)
    x = torch.randn(1, tokens, dim, device=dev(), generator=torch.Generator(device=dev()).manual_seed(tokens)).bfloat16()
    weight = lambda m: (m.weight.double(), m.bias.double())
    with torch.no_grad():
        want = F.linear(F.gelu(F.linear(x.double(), *weight(ffn[0])), approximate="tanh"), *weight(ffn[2]))
        rel = lambda y: float((y.double() - want).norm() / want.norm())
        # one rounding to bf16 (2^-9 of a value, 1.7e-3 root mean square) less in the hidden values.  One row has few values: their
        # distances scatter by some percent about the same mean
        assert rel(feed_forward(ffn, x)) <= rel(ffn(x)) * (1.1 if tokens == 1 else 1.0)


@pytest.mark.gpu
@pytest.mark.parametrize("what", ["hook", "pre-hook", "hook of all modules", "own forward", "other weight", "one more module", "exact gelu"])
def test_what_hangs_on_the_modules_is_seen(monkeypatch, what):
    from worldattention_b200.causal_dit import feed_forward
    ffn = _ffn().to(dev(), torch.bfloat16)
    x = torch.randn(1, 40, 256, device=dev()).bfloat16()
    seen = []
    handle = None
    if what == "hook":
        handle = ffn[1].register_forward_hook(lambda *a: seen.append(1))
    elif what == "pre-hook":
        handle = ffn.register_forward_pre_hook(lambda *a: seen.append(1))
    elif what == "hook of all modules":
        handle = nn.modules.module.register_module_forward_hook(lambda m, *a: seen.append(1) if m is ffn[1] else None)
    elif what == "own forward":
        monkeypatch.setattr(ffn[0], "forward", lambda t: seen.append(1) or F.linear(t, ffn[0].weight, ffn[0].bias))
    elif what == "other weight":
        plain = ffn[0].weight.detach().clone()
        del ffn[0].weight
        ffn[0].weight = plain
    elif what == "one more module":
        ffn.append(nn.Dropout(0.0))
    else:
        ffn[1] = nn.GELU()
    try:
        with torch.no_grad():
            got = feed_forward(ffn, x)
            assert len(seen) == (what not in ("other weight", "one more module", "exact gelu"))
            assert torch.equal(got, ffn(x))
    finally:
        if handle is not None:
            handle.remove()


@pytest.mark.gpu
def test_no_tokens_autocast_and_forward_mode():
    from worldattention_b200.causal_dit import feed_forward
    ffn = _ffn().to(dev(), torch.bfloat16)
    x = torch.randn(1, 40, 256, device=dev()).bfloat16()
    with torch.no_grad():
        assert feed_forward(ffn, x[:, :0]).shape == (1, 0, 256)
        with torch.autocast("cuda", torch.float16):
            assert feed_forward(ffn, x).dtype == ffn(x).dtype == torch.float16
        y, dy = torch.func.jvp(ffn, (x,), (x,))
        assert torch.equal(y, ffn(x)) and dy.shape == y.shape and bool(dy.any())
