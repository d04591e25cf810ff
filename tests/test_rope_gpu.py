"""The fused q/k RMSNorm + causal rotary embedding kernel against the numpy oracle and the reference's own outputs."""
import numpy as np
import pytest
import torch

from oracle import rope_oracle as R
from tests.helpers import dev, to_gpu, to_np

pytestmark = pytest.mark.gpu


def test_norm_and_rope_match_oracle_and_reference(golden):
    from worldattention_b200 import rope
    g = golden("qk_norm_rope")
    grid, start, eps = tuple(int(v) for v in g["grid"]), int(g["start_frame"]), float(g["eps"])
    freqs = torch.from_numpy(g["freqs"])
    for tag, one_step in (("fp32", 0.0), ("bf16", 2 ** -7)):
        x = to_gpu(g[f"x_{tag}"], tag)
        w = to_gpu(g[f"weight_{tag}"], tag)
        got = rope.qk_norm_rope(x, w, eps, [grid], freqs, start, heads=2)
        want = R.qk_norm_rope(g[f"x_{tag}"], g[f"weight_{tag}"], eps, grid, g["freqs"], start, 2, tag)
        assert np.array_equal(to_np(got), want)                               # same arithmetic as the oracle, bit for bit
        ref = g[f"roped_{tag}"]                                              # the reference's own output
        if tag == "fp32":
            np.testing.assert_allclose(to_np(got), ref, rtol=0, atol=5e-6)
        else:       # torch's float32 mean may put a normalised value one bf16 step away; the rotation mixes a pair
            np.testing.assert_allclose(to_np(got), ref, rtol=0, atol=2 * one_step * np.abs(ref).max())
            assert np.mean(to_np(got) != ref) < 5e-3
        # rotation alone, the reference's signature; float64 product stored once: identical to the reference
        only = rope.causal_rope_apply(x.view(1, -1, 2, 128), torch.tensor([grid]), freqs, start_frame=start)
        assert np.array_equal(to_np(only), g[f"rope_only_{tag}"])
    # strided input (a slice of a fused q/k/v projection) and a frame offset beyond the table are handled
    qkv = torch.randn(1, 24, 3 * 256, device=dev()).bfloat16()
    q = qkv[..., :256]
    a = rope.qk_norm_rope(q, to_gpu(g["weight_bf16"], "bf16"), eps, [grid], freqs, start, heads=2)
    b = rope.qk_norm_rope(q.contiguous(), to_gpu(g["weight_bf16"], "bf16"), eps, [grid], freqs, start, heads=2)
    assert torch.equal(a, b)
    with pytest.raises(NotImplementedError):
        rope.causal_rope_apply(x.view(1, -1, 2, 128), torch.tensor([[1, 3, 4]]), freqs)


def _awkward(x):
    """Rows of zeros, subnormals, the largest and smallest values, infinities and NaN among the ordinary ones."""
    rows = x.view(-1, x.shape[-1])
    for i, value in enumerate((0.0, 1e-39, 3e38, 1e-30, 1e25, float("inf"), float("nan"))):
        if 2 * i + 1 < rows.shape[0]:
            rows[2 * i] = value
            rows[2 * i + 1, i::7] = value
    return x


@pytest.mark.parametrize("batch,grid,heads,d", [(1, (1, 1, 1), 1, 8), (2, (1, 3, 5), 2, 128), (1, (3, 7, 11), 12, 128), (1, (2, 9, 13), 16, 128),
                                                (1, (2, 5, 4), 12, 64), (3, (1, 4, 4), 5, 256), (1, (1, 2, 17), 24, 32)])
def test_bf16_rows_match_the_float64_rotation_bit_for_bit(batch, grid, heads, d):
    """bf16 weights take the kernel that rotates in float32 where that settles the result; the same weights in float32, and
    heads that do not lie side by side, take the float64 ones."""
    from worldattention_b200 import rope
    from worldattention_b200.causal_dit import rope_table
    n = grid[0] * grid[1] * grid[2]
    g = torch.Generator(device=dev()).manual_seed(d + heads)
    freqs = rope_table(d) if d >= 32 else torch.polar(torch.ones(64, d // 2, dtype=torch.float64), torch.randn(64, d // 2, dtype=torch.float64))
    w = (1 + 0.3 * torch.randn(heads * d, generator=g, device=dev())).bfloat16()
    start = torch.full((1,), 11, dtype=torch.int32, device=dev())
    for awkward in (False, True):
        x = torch.randn(batch, n, heads * d, generator=g, device=dev()).bfloat16()
        x = _awkward(x) if awkward else x
        same = lambda a, b: torch.equal(a.contiguous().view(torch.int16), b.contiguous().view(torch.int16))
        for frame in (0, start):
            got = rope.qk_norm_rope(x, w, 1e-6, grid, freqs, frame, heads=heads)
            assert same(got, rope.qk_norm_rope(x, w.float(), 1e-6, grid, freqs, frame, heads=heads))
        assert same(rope.qk_norm_rope(x, w, 1e-6, None, None, heads=heads), rope.qk_norm_rope(x, w.float(), 1e-6, None, None, heads=heads))
        x4 = x.view(batch, n, heads, d)
        spread = torch.empty(batch, n, heads, d + 2, dtype=x.dtype, device=dev())[..., :d].copy_(x4)
        assert same(rope.causal_rope_apply(x4, grid, freqs, 5), rope.causal_rope_apply(spread, grid, freqs, 5))


def test_factors_below_float32_are_rotated_in_float64():
    """A table's smallest factors times the largest values: what float32 cannot hold of the factor is not in the rotation's bound."""
    from worldattention_b200 import rope
    g = torch.Generator(device=dev()).manual_seed(7)
    n, heads, d = 12, 2, 128
    sign = torch.randn(64, d // 2, 2, generator=g, device=dev(), dtype=torch.float64)
    freqs = torch.view_as_complex(sign * 2.0 ** torch.randint(-170, -90, (64, d // 2, 2), generator=g, device=dev()).double()).cpu()
    freqs[:, ::3] = freqs[:, ::3].imag * 1j + 1.0
    x = (torch.randn(1, n, heads, d, generator=g, device=dev()) * 2.0 ** torch.randint(0, 120, (1, n, heads, d), generator=g, device=dev()).float()).bfloat16()
    x[..., 1::4] = 0
    spread = torch.empty(1, n, heads, d + 2, dtype=x.dtype, device=dev())[..., :d].copy_(x)
    got, want = (rope.causal_rope_apply(t, (3, 2, 2), freqs, 5) for t in (x, spread))
    assert torch.equal(got.contiguous().view(torch.int16), want.contiguous().view(torch.int16))
