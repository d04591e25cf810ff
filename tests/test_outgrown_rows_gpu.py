"""Rows whose later key blocks outgrow the reference point that the tcgen05 kernel took from an earlier one, and the work order of
calls whose keys and values are more than L2 keeps, both against the library's float32 path."""
import pytest
import torch

from tests.helpers import attention_error, dev, to_np

pytestmark = pytest.mark.gpu
D = 128
MAX_ABS, MEAN_REL = 2e-2, 1e-2      # as for the other calls (bf16 operands and result, values of unit variance)


# 128-token blocks; 64-token blocks, one query block per work item and two.  A step of 3 stays below what makes a row look again, 20
# does not, and 200 is beyond the range of the exponential.
@pytest.mark.parametrize("block,heads,nq", [(128, 3, 2), (64, 3, 2), (64, 24, 8)])
@pytest.mark.parametrize("step", [3.0, 20.0, 200.0])
def test_later_blocks_outgrow_earlier_ones(block, heads, nq, step):
    from worldattention_b200.hsa.branches import hsa_partials
    g = torch.Generator(device=dev()).manual_seed(block + heads)
    draw = lambda n: torch.randn(1, n, heads, D, generator=g, device=dev())
    nkv, slots = 9, 300
    q, k, v, kc, vc = draw(nq * block - 5) * 0.3, draw(nkv * block - 17) * 0.3, draw(nkv * block - 17), draw(slots) * 0.3, draw(slots)
    # logits in powers of two: `step` per block for most rows, the same downwards for every third
    q[..., 0] = 8.0
    q[:, ::3, :, 0] = -8.0
    unit = step / (8.0 * D ** -0.5 * 1.4426950408889634)
    k[..., 0] = (torch.arange(k.shape[1], device=dev()) // block)[None, :, None] * unit
    kc[..., 0] = (torch.arange(slots, device=dev()) // 100)[None, :, None] * unit
    args = [t.bfloat16() for t in (q, k, v, kc, vc)]
    index = torch.arange(nkv, dtype=torch.int32, device=dev()).expand(1, heads, nq, nkv).contiguous()
    num = torch.full((1, heads, nq), nkv, dtype=torch.int32, device=dev())
    num[0, 0, 0] = 4
    got, want = (hsa_partials(*args, index, num, block, force_generic=generic) for generic in (False, True))
    assert got[4] and not want[4]
    for a, b in zip(got[:4], want[:4]):
        a, b = to_np(a), to_np(b)
        max_abs, mean_rel = attention_error(a, b)
        assert max_abs < max(MAX_ABS, 1e-5 * abs(b).max()) and mean_rel < MEAN_REL      # the normalisers reach a thousand


def _lists(heads, nq, nkv, own):
    """Every query block takes all key blocks in order; with `own` the even ones the even blocks, the odd ones the odd blocks."""
    index = torch.arange(nkv, dtype=torch.int32, device=dev()).expand(1, heads, nq, nkv).contiguous()
    num = torch.full((1, heads, nq), nkv, dtype=torch.int32, device=dev())
    if own:
        half = nkv // 2
        index[:, :, 0::2, :half] = torch.arange(0, 2 * half, 2, dtype=torch.int32, device=dev())
        index[:, :, 1::2, :half] = torch.arange(1, 2 * half, 2, dtype=torch.int32, device=dev())
        num[:] = half
    return index, num


# 128-token blocks; 64-token blocks, one query block per work item; two that share their key blocks; two that share none (a tile then
# has 64 keys for either).
SHAPES = [(128, 3, 2, False), (64, 3, 2, False), (64, 24, 8, False), (64, 24, 8, True)]


# Powers of two that each tile's keys lie above the ones before.  A reference point moves where the growth since then exceeds about 8;
# more than 12 in one tile make the next tile look for its maximum first, whether it grows or not.
STEPS = {"once in a while": [9, 0, 0, 60, 3, 11, 0, 13, 0, 0, 0, 9], "steep, then flat": [100, 0, 100, 100, 0, 0, 73, 71, 0, 200, 0, 0],
         "up and down": [80, -80, 160, -100, 30, -200, 300, -5, 10, 64, 8, 1], "down": [-90, -3, -200, 0, 0, -10, 0, 0, 0, 0, 0, 0]}


@pytest.mark.parametrize("block,heads,nq,own", SHAPES)
@pytest.mark.parametrize("steps", list(STEPS))
def test_growth_that_comes_and_goes(block, heads, nq, own, steps):
    from worldattention_b200.hsa.branches import hsa_partials
    g = torch.Generator(device=dev()).manual_seed(block + heads + own)
    draw = lambda n: torch.randn(1, n, heads, D, generator=g, device=dev())
    level = torch.cumsum(torch.tensor([0] + STEPS[steps], device=dev(), dtype=torch.float32), 0)
    tile = max(128 // block, 1)               # blocks of a tile
    nkv, slots = 13 * tile, 13 * 128
    q, k, v, kc, vc = draw(nq * block - 5) * 0.3, draw(nkv * block - 17) * 0.3, draw(nkv * block - 17), draw(slots - 17) * 0.3, draw(slots - 17)
    q[..., 0] = 8.0
    unit = 1 / (8.0 * D ** -0.5 * 1.4426950408889634)
    k[..., 0] = (level[torch.arange(k.shape[1], device=dev()) // 128] * unit)[None, :, None]
    kc[..., 0] = (level[torch.arange(kc.shape[1], device=dev()) // 128] * unit)[None, :, None]
    args = [t.bfloat16() for t in (q, k, v, kc, vc)]
    index, num = _lists(heads, nq, nkv, own)
    got, want = (hsa_partials(*args, index, num, block, force_generic=generic) for generic in (False, True))
    assert got[4] and not want[4]
    for a, b in zip(got[:4], want[:4]):
        a, b = to_np(a), to_np(b)
        max_abs, mean_rel = attention_error(a, b)
        assert max_abs < max(MAX_ABS, 1e-5 * abs(b).max()) and mean_rel < MEAN_REL


# ONE key of the second tile lies `nats` above all others, for every row alike: nothing but the exponential of its own column can tell.
# Columns 0..7 of every 64 are computed by a polynomial, the others by the special-function unit; 88 nats are 127 powers of two, from
# 90 on float32 overflows, and 177, 266 and 355 are 256, 384 and 512 powers of two.
@pytest.mark.parametrize("block,heads,nq,own", SHAPES)
@pytest.mark.parametrize("nats", [60.0, 88.0, 90.0, 140.0, 177.4, 200.0, 265.0, 355.0, 450.0])
def test_one_key_outgrows_the_rest(block, heads, nq, own, nats):
    from worldattention_b200.hsa.branches import hsa_partials
    g = torch.Generator(device=dev()).manual_seed(block + heads + own)
    draw = lambda n: torch.randn(1, n, heads, D, generator=g, device=dev())
    nkv, slots = 9, 300
    q, k, v, kc, vc = draw(nq * block - 5) * 0.3, draw(nkv * block - 17) * 0.3, draw(nkv * block - 17), draw(slots) * 0.3, draw(slots)
    q[..., 0] = 16.0
    k[..., 0] = kc[..., 0] = 0.0
    index, num = _lists(heads, nq, nkv, own)
    for column in (0, 3, 7, 8) if own else (0, 3, 7, 8, 64, 71, 72):
        k2, kc2 = k.clone(), kc.clone()
        for token in (128 + column, 192 + column) if own else (128 + column,):
            k2[:, token, :, 0] = nats / (16.0 * D ** -0.5)
        kc2[:, 128 + column, :, 0] = nats / (16.0 * D ** -0.5)
        args = [t.bfloat16() for t in (q, k2, v, kc2, vc)]
        got, want = (hsa_partials(*args, index, num, block, force_generic=generic) for generic in (False, True))
        assert got[4] and not want[4]
        for a, b in zip(got[:4], want[:4]):
            a, b = to_np(a), to_np(b)
            max_abs, mean_rel = attention_error(a, b)
            assert max_abs < max(MAX_ABS, 1e-5 * abs(b).max()) and mean_rel < MEAN_REL, column


@pytest.mark.parametrize("block,heads,nq,own", SHAPES)
@pytest.mark.parametrize("column", [0, 7, 8, 130, 135, 140])      # of the first tile and of the second
def test_a_key_that_is_no_number_reaches_the_rows_that_chose_it(block, heads, nq, own, column):
    from worldattention_b200.hsa.branches import hsa_partials
    g = torch.Generator(device=dev()).manual_seed(column)
    draw = lambda n: torch.randn(1, n, heads, D, generator=g, device=dev())
    nkv = 9
    q, k, v, kc, vc = (t.bfloat16() for t in (draw(nq * block - 5), draw(nkv * block - 17), draw(nkv * block - 17), draw(70), draw(70)))
    k[:, column, 0, 3] = float("nan")
    index, num = _lists(heads, nq, nkv, own)
    got, want = (hsa_partials(q, k, v, kc, vc, index, num, block, force_generic=generic)[0].isnan() for generic in (False, True))
    assert bool(want[:, :block, 0].all()) and torch.equal(got, want)


@pytest.mark.parametrize("heads,q_blocks,kv", [(12, 13, 11003), (5, 75, 30000), (24, 7, 6000)])
def test_every_item_of_a_call_ordered_by_heads_is_done(heads, q_blocks, kv):
    from worldattention_b200.hsa import hsa_attention
    assert heads * q_blocks > torch.cuda.get_device_properties(0).multi_processor_count and 4 * heads * kv * D > 64 << 20
    g = torch.Generator(device=dev()).manual_seed(kv)
    draw = lambda n: torch.randn(1, n, heads, D, generator=g, device=dev())
    q, k, v, kc, vc = (t.bfloat16() for t in (draw(q_blocks * 64 - 9) * 0.5, draw(kv) * 0.5, draw(kv), draw(60), draw(60)))
    kwargs = dict(k_coarse=kc, v_coarse=vc, k_proj_mat=None, v_proj_mat=None, block_size=64)
    out, (_, num, _, used) = hsa_attention(q, k, v, return_routing=True, check_status=True, **kwargs)
    want, (_, num_g, _, used_g) = hsa_attention(q, k, v, return_routing=True, force_generic=True, **kwargs)
    assert used and not used_g and torch.equal(num, num_g)
    max_abs, mean_rel = attention_error(to_np(out), to_np(want))
    assert max_abs < 2 * 2 ** -6 and mean_rel < MEAN_REL      # |v| < 4 of a mean of hundreds: a step of bf16 each way
