"""The output head's norm and modulation: in one launch only where that is what the modules compute."""
import pytest
import torch

from tests.helpers import dev


def _model(dim=256, **kw):
    from worldattention_b200.causal_dit import CausalDiT, DiTConfig
    torch.manual_seed(0)
    return CausalDiT(DiTConfig(dim=dim, heads=2, ffn_dim=64, layers=1, text_dim=64, latent_hw=(6, 10), **kw))


def _inputs(model, frames=3):
    x = torch.randn(1, frames * 15, model.cfg.dim) * 2 + 0.3
    return [t.to(dev()).bfloat16() for t in (x, torch.randn(1, frames, 1, model.cfg.dim) * 0.3, torch.randn(1, frames, 1, model.cfg.dim))]


def _plain(model, x, scale, shift):
    return (model.head_norm(x).unflatten(1, (scale.shape[1], 15)) * (1 + scale) + shift).flatten(1, 2)


def test_latents_of_another_size_are_refused():
    model = _model().eval()
    x, e = torch.randn(1, 60, 256), torch.randn(1, 3, 1, 256)
    with pytest.raises(RuntimeError):
        model._modulated(x, e, e)


@pytest.mark.gpu
@pytest.mark.parametrize("dim", [256, 1544, 4096])
def test_distance_from_float64_is_that_of_the_expressions(dim):
    model = _model(dim).to(dev(), torch.bfloat16)
    x, scale, shift = _inputs(model)
    with torch.no_grad():
        got, plain = model._modulated(x, scale, shift), _plain(model, x, scale, shift)
        xd = x.double()
        want = (xd - xd.mean(-1, keepdim=True)) / (xd.var(-1, unbiased=False, keepdim=True) + 1e-6).sqrt()
        want = (want.unflatten(1, (3, 15)) * (1 + scale.double()) + shift.double()).flatten(1, 2)
        rel = lambda y: float((y.double() - want).norm() / want.norm())
        # the same rounding points; a float32 statistic summed in another order moves one value in some thousand to its neighbour
        assert rel(got) <= rel(plain) * 1.001 and float((got != plain).float().mean()) < 1e-3


@pytest.mark.gpu
@pytest.mark.parametrize("what", ["hook", "hook of all modules", "affine norm", "other norm", "blocks as expressions", "wide rows"])
def test_what_the_launch_does_not_compute_goes_through_the_modules(what):
    from worldattention_b200.causal_dit import _LayerNorm
    model = _model(4104 if what == "wide rows" else 256).to(dev(), torch.bfloat16)
    x, scale, shift = _inputs(model)
    seen, handle = [], None
    if what == "hook":
        handle = model.head_norm.register_forward_hook(lambda *a: seen.append(1))
    elif what == "hook of all modules":
        handle = torch.nn.modules.module.register_module_forward_hook(lambda *a: seen.append(1))
    elif what == "affine norm":
        model.head_norm = _LayerNorm(256, 1e-6, elementwise_affine=True).to(dev(), torch.bfloat16)
        torch.nn.init.normal_(model.head_norm.weight)
    elif what == "other norm":
        model.head_norm = torch.nn.Identity()
    else:
        for blk in model.blocks:
            blk.fused = False
    try:
        with torch.no_grad():
            got = model._modulated(x, scale, shift)
            assert len(seen) == ("hook" in what) and torch.equal(got, _plain(model, x, scale, shift))
    finally:
        if handle is not None:
            handle.remove()


@pytest.mark.gpu
@pytest.mark.parametrize("frames,h,w", [(3, 60, 104), (1, 18, 30), (2, 2, 2), (3, 26, 34)])
def test_patch_embedding_in_channels_last_order(frames, h, w):
    """Latents laid channels last go through the same convolution: no further from float64 than in their own order."""
    conv = _model(1536).patch_embedding.to(dev(), torch.bfloat16)
    latents = torch.randn(1, frames, 16, h, w, device=dev(), generator=torch.Generator(device=dev()).manual_seed(h)).bfloat16().permute(0, 2, 1, 3, 4)
    with torch.no_grad():
        plain, got = conv(latents), conv(latents.contiguous(memory_format=torch.channels_last_3d))
        want = torch.nn.functional.conv3d(latents.double(), conv.weight.double(), conv.bias.double(), stride=(1, 2, 2))
    rel = lambda y: float((y.double() - want).norm() / want.norm())
    # 64 products per value in float32, rounded to bf16 once: another order of the sums moves one value in some thousand
    assert rel(got) <= rel(plain) * 1.001
    assert got.flatten(2).transpose(1, 2).is_contiguous()
