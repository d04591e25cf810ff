"""What `wa_hsa_forward` asks its caller to set aside (no GPU needed): the bf16 copy of float32 keys and values is in it for the calls that
make one, and for no others."""
import ctypes

import pytest

B, H, D = 1, 12, 128


def _bytes(q_len, kv_len, block=64, k_stride=H * D, k_ptr=1 << 20, **fields):
    from worldattention_b200 import _lib
    p = _lib.HsaParams(B=B, H=H, D=D, Lq=q_len, Lkv=kv_len, Lc=100, block_size=block)
    row = lambda stride, ptr=1 << 20: _lib.Tensor4(ptr=ptr, dtype=0, stride_b=kv_len * stride, stride_l=stride, stride_h=D)
    p.q = p.v = p.k_coarse = p.v_coarse = p.out = row(H * D)
    p.k = row(k_stride, k_ptr)
    for name, value in fields.items():
        setattr(p, name, value)
    return _lib.lib().wa_hsa_workspace_bytes(ctypes.byref(p))


@pytest.mark.parametrize("q_len,kv_len,block", [(1560, 4680, 64), (4680, 12480, 128), (390, 1170, 64)])
def test_room_for_rounded_keys_where_they_are_rounded(q_len, kv_len, block):
    rounded = 2 * 2 * B * kv_len * H * D if B * H * -(-q_len // block) >= 148 else 0
    plain = _bytes(q_len, kv_len, block, k_stride=H * D + 2)                       # rows that are not 16-byte aligned are not rounded
    assert _bytes(q_len, kv_len, block, k_ptr=(1 << 20) + 4) == plain
    assert _bytes(q_len, kv_len, block) == plain + rounded
    assert _bytes(q_len, kv_len, block, part_sparse=1 << 20) == plain              # nor are those of a call with partial outputs
    assert _bytes(q_len, kv_len, block, k_stride=0, k_ptr=0) == plain + rounded    # not known yet: enough for either


# fixed counts and a caller's own routing select no more of a longer cache; the room for the copy is bounded by 512 MB
@pytest.mark.parametrize("kv_len,fields,expected", [
    (16384, dict(topk_per_head=1 << 20), True), (16385, dict(topk_per_head=1 << 20), False), (748800, dict(topk_per_head=1 << 20), False),
    (16384, dict(index_in=1 << 20, num_in=1 << 20), True), (16385, dict(index_in=1 << 20, num_in=1 << 20), False),
    (16385, {}, True), ((512 << 20) // (4 * H * D), {}, True), ((512 << 20) // (4 * H * D) + 1, {}, False), (748800, {}, False)])
def test_long_caches_are_rounded_where_that_pays(kv_len, fields, expected):
    assert _bytes(4680, kv_len, **fields) - _bytes(4680, kv_len, k_stride=H * D + 2, **fields) == (4 * B * kv_len * H * D + 255) // 256 * 256 * expected
