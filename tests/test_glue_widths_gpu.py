"""The block glue's kernels at the row lengths where a lane's share of a row changes, against the tensor expressions."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("c", [8, 248, 512, 520, 1024, 1032, 1536, 1544, 2048, 2056, 4096, 8200])
def test_rows_of_every_width(c):
    from worldattention_b200.causal_dit import _LayerNorm, gated_residual, ln_modulate
    dev = torch.device("cuda:0")
    g = torch.Generator(device=dev).manual_seed(c)
    frames, tokens = 3, 11
    x = (torch.randn(1, frames * tokens, c, generator=g, device=dev) * 2 + 0.3).bfloat16()
    y = torch.randn(1, frames * tokens, c, generator=g, device=dev).bfloat16()
    e = (torch.randn(1, frames, 3, c, generator=g, device=dev) * 0.5).bfloat16().chunk(3, dim=2)
    want = x + (y.unflatten(1, (frames, tokens)) * e[2]).flatten(1, 2)
    assert torch.equal(gated_residual(x, y, e[2], tokens_per_frame=tokens), want)
    assert torch.equal(gated_residual(x, y), x + y)
    if c > 4096:
        with pytest.raises(NotImplementedError):
            ln_modulate(x, 1e-6)
        return
    want = (_LayerNorm(c, 1e-6).to(dev)(x).unflatten(1, (frames, tokens)) * (1 + e[1]) + e[0]).flatten(1, 2).float()
    diff = (ln_modulate(x, 1e-6, scale=e[1], shift=e[0], tokens_per_frame=tokens).float() - want).abs()
    # the same rounding points; float32 statistics in another order put a normalised value at most one bf16 step away, whose
    # product with 1 + scale (below 4 here) is rounded again: two steps of the largest value
    assert float(diff.max()) <= 2 * 2 ** -8 * float(want.abs().max()) and float((diff > 0).float().mean()) < 0.02


def test_a_modulation_holds_a_vector_for_every_frame():
    """The kernels take the vector of row / tokens_per_frame: rows behind the last frame are refused, not read with what lies there."""
    from worldattention_b200.causal_dit import gated_residual, ln_modulate
    dev = torch.device("cuda:0")
    x, e = torch.randn(1, 33, 64, device=dev).bfloat16(), torch.randn(1, 3, 1, 64, device=dev).bfloat16()
    for tokens in (10, 1):
        for call in (lambda: ln_modulate(x, 1e-6, scale=e, tokens_per_frame=tokens), lambda: ln_modulate(x, 1e-6, shift=e, tokens_per_frame=tokens),
                     lambda: gated_residual(x, x, e, tokens_per_frame=tokens)):
            with pytest.raises(ValueError, match="frames"):
                call()
    with pytest.raises(ValueError, match="modulation"):
        gated_residual(x, x, e[..., :56], tokens_per_frame=11)
    gated_residual(x, x, e, tokens_per_frame=11)
    gated_residual(x, x, e, tokens_per_frame=40)             # frames that no row reaches
