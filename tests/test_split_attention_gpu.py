"""The float32-exact attention on matrix instructions (head_dim 128) against float64 softmax attention.

Every product is a sum of exact bf16 products accumulated in float32, so a result is off by the float32 accumulation of the
scores (128 terms, |s| up to a few units) and of P V: a few 1e-6 of the largest value.  The bound of the first tests is 2e-5 of
that, which a probability or an operand kept in 16 bits (2^-9) would miss by two orders; the last ones look for products left
out and for sums that lose the same way at every step."""
import numpy as np
import pytest
import torch

from tests.helpers import dev

pytestmark = pytest.mark.gpu
D = 128


def _exact(q, k, v, keys_of_row):
    """float64 attention of `[L, H, D]` tensors; `keys_of_row(head, row)` gives the key ids a query row sees."""
    q, k, v = (t.double().cpu().numpy() for t in (q, k, v))
    out = np.zeros(q.shape)
    for h in range(q.shape[1]):
        for r in range(q.shape[0]):
            ids = keys_of_row(h, r)
            if len(ids) == 0:
                continue
            s = k[ids, h] @ q[r, h] / np.sqrt(D)
            p = np.exp(s - s.max())
            out[r, h] = p @ v[ids, h] / p.sum()
    return out


def _sparse(q, k, v, index, num, block):
    """The C entry with rounded inputs and an unrounded float32 result."""
    from worldattention_b200 import _lib
    out = torch.empty(q.shape, device=q.device, dtype=torch.float32)
    _lib.check(_lib.lib().wa_block_sparse_forward(
        _lib.t4_bhnd(q), _lib.t4_bhnd(k), _lib.t4_bhnd(v), _lib.t4_bhnd(out), 1, q.shape[1], q.shape[2], k.shape[2], D, block,
        index.data_ptr(), num.data_ptr(), index.shape[-1], None, 1, 0, None, _lib.stream_ptr(q.device)))
    return out


def _linear(q, kc, vc, lse=None):
    from worldattention_b200 import _lib
    out = torch.empty(q.shape, device=q.device, dtype=torch.float32)
    _lib.check(_lib.lib().wa_linear_branch(_lib.t4_blhd(q), _lib.t4_blhd(kc), _lib.t4_blhd(vc), _lib.t4_blhd(out), 1, q.shape[2], q.shape[1],
                                           kc.shape[1], D, 0, _lib.ptr(lse), _lib.stream_ptr(q.device)))
    return out


@pytest.mark.parametrize("block,lq,lkv,dtype", [(64, 130, 321, "fp32"), (100, 205, 333, "fp32"), (16, 40, 75, "bf16"), (128, 129, 1, "bf16"),
                                                (1, 3, 70, "fp32")])
def test_block_sparse_branch(block, lq, lkv, dtype):
    g = torch.Generator(device=dev()).manual_seed(lq)
    heads, nq, nkv = 2, -(-lq // block), -(-lkv // block)
    make = lambda n: torch.randn((1, heads, n, D), generator=g, device=dev()).to(torch.float32 if dtype == "fp32" else torch.bfloat16)
    q, k, v = make(lq), make(lkv), make(lkv)
    index = torch.stack([torch.randperm(nkv, generator=g, device=dev()) for _ in range(heads * nq)]).view(1, heads, nq, nkv).int()
    num = torch.randint(0, nkv + 1, (1, heads, nq), generator=g, device=dev()).int()
    num[0, 0, 0], num[0, 1, -1] = nkv, 0                  # everything, and nothing
    out = _sparse(q, k, v, index, num, block)
    rounded = [t.to(torch.bfloat16).float()[0].transpose(0, 1) for t in (q, k, v)]      # the branch takes bf16 values
    def keys(h, r):
        chosen = index[0, h, r // block, : int(num[0, h, r // block])].tolist()
        return [t for b in chosen for t in range(b * block, min((b + 1) * block, lkv))]
    want = _exact(*rounded, keys)
    got = out[0].transpose(0, 1).double().cpu().numpy()
    assert np.abs(got - want).max() <= 2e-5 * max(np.abs(want).max(), 1e-3)


@pytest.mark.parametrize("lq,lc,scale", [(65, 1, 1.0), (64, 33, 1.0), (200, 75, 1.0), (31, 160, 4.0)])
def test_linear_branch_float32(lq, lc, scale):
    g = torch.Generator(device=dev()).manual_seed(lc)
    q, kc, vc = (torch.randn((1, n, 3, D), generator=g, device=dev()) * s for n, s in ((lq, scale), (lc, 1.0), (lc, 1.0)))
    got = _linear(q, kc, vc)[0].double().cpu().numpy()
    want = _exact(q[0], kc[0], vc[0], lambda h, r: list(range(lc)))
    # scores of size s carry an absolute float32 error of about s * 2^-22: it multiplies the probabilities
    assert np.abs(got - want).max() <= 2e-5 * scale * np.abs(want).max()


def test_strided_rows_and_infinities():
    # rows of a wider tensor; an infinite value stays infinite (and of its sign)
    g = torch.Generator(device=dev()).manual_seed(3)
    wide = torch.randn((1, 70, 3, 2 * D), generator=g, device=dev())
    q, kc, vc = wide[:, :40, :, :D], wide[..., D:], torch.randn((1, 70, 3, D), generator=g, device=dev())
    vc[0, 7, 1, 9] = -float("inf")
    got, plain = _linear(q, kc, vc), _linear(q.contiguous(), kc.contiguous(), vc)
    assert torch.equal(got.nan_to_num(), plain.nan_to_num())
    assert bool((got[0, :, 1, 9] == -float("inf")).all())
    got[0, :, 1, 9] = 0
    assert bool(torch.isfinite(got).all())


def test_every_partial_product_of_a_score_counts():
    # parts 1, 2^-7 - 2^-15 and 2^-15 - 2^-23: the products of the second and third ones are 2^-21 of the whole
    q = torch.full((1, 64, 1, D), 1 + 2.0 ** -7 - 2.0 ** -23, device=dev())
    lse = torch.empty((1, 1, 64), device=dev())
    _linear(q, q[:, :1].contiguous(), q[:, :1].contiguous(), lse)          # one slot: the score itself
    want = float(q[0, 0, 0, 0].double()) ** 2 * np.sqrt(D)
    # eight 16-term sums, each cut by 2^-23 at most, added up with 4.5 roundings of the whole (n / 8 at the n-th), one for the scale
    assert float((lse.double() / want - 1).abs().max()) <= 2.0 ** -23 + 5.5 * 2.0 ** -24


@pytest.mark.parametrize("keys,rounded", [(4680, True), (2000, False)])
def test_long_rows_of_one_sign_lose_nothing(keys, rounded):
    g = torch.Generator(device=dev()).manual_seed(keys)
    q, k, v = (torch.randn((1, 2, n, D), generator=g, device=dev()) for n in (128, keys, keys))
    v = v.abs()
    if rounded:
        block = 64
        nkv = -(-keys // block)
        index = torch.arange(nkv, device=dev(), dtype=torch.int32).expand(1, 2, 2, nkv).contiguous()
        got = _sparse(q, k, v, index, torch.full((1, 2, 2), nkv, device=dev(), dtype=torch.int32), block)
        q, k, v = (t.to(torch.bfloat16) for t in (q, k, v))
    else:
        got = _linear(*(t.transpose(1, 2).contiguous() for t in (q, k, v))).transpose(1, 2)
    s = q[0].double() @ k[0].double().transpose(1, 2) / np.sqrt(D)
    want = torch.softmax(s, -1) @ v[0].double()
    # a step of 16 keys is cut by 2^-23 per leading product, always downward; everything else rounds either way
    assert abs(float((got[0].double() / want - 1).mean())) <= 3 * 2.0 ** -23


@pytest.mark.parametrize("hidden", [8, 16, 32, 40])
def test_leading_keys_without_weight(hidden):
    # the first `hidden` keys score -inf: they have no weight, whatever chunk of keys they fill; a row of nothing else is NaN
    g = torch.Generator(device=dev()).manual_seed(hidden)
    q, kc, vc = (torch.randn((1, n, 2, D), generator=g, device=dev()) for n in (20, 70, 70))
    q[..., 5] = 1.0
    kc[:, :hidden, :, 5] = -float("inf")
    want = _exact(q[0], kc[0, hidden:], vc[0, hidden:], lambda h, r: list(range(70 - hidden)))
    got = _linear(q, kc, vc)[0].double().cpu().numpy()
    assert np.abs(got - want).max() <= 2e-5 * np.abs(want).max()
    assert bool(torch.isnan(_linear(q, kc[:, :hidden], vc[:, :hidden])).all())


@pytest.mark.parametrize("bits", [0x7f800001, 0x7fc00000, -0x7fffff])    # the first and last (0xff800001) are infinities in their upper halves
def test_every_nan_stays_one(bits):
    g = torch.Generator(device=dev()).manual_seed(1)
    q, kc, vc = (torch.randn((1, n, 2, D), generator=g, device=dev()) for n in (20, 40, 40))
    q.view(torch.int32)[0, 3, 1, 7] = bits
    vc.view(torch.int32)[0, 9, 0, 5] = bits
    nan = torch.isnan(_linear(q, kc, vc))
    want = torch.zeros_like(nan)
    want[0, 3, 1], want[0, :, 0, 5] = True, True
    assert torch.equal(nan, want)
