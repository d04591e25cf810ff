"""The native host module's own work: what it refuses, how it reads its arguments, and the workspaces it keeps."""
import sys
import threading
import time

import numpy as np
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


def test_integers_of_other_types():
    options = _inputs()

    class Size:
        def __int__(self):
            return token

    token = int("1000064")          # an object of its own, so that references to it can be counted
    want = _attend(**options)
    for as_given in (np.int64(64), 64.0, torch.tensor(64)):
        assert torch.equal(_attend(**{**options, "block_size": as_given}), want)
    before = sys.getrefcount(token)
    for _ in range(5):
        _attend(**{**options, "proj_segment_len": Size(), "k_pooled_valid": Size()})      # both larger than what they bound
    assert sys.getrefcount(token) == before
    with pytest.raises(TypeError):
        _attend(**{**options, "block_size": "sixty-four".encode})


def test_modulation_with_and_without_the_token_axis():
    from worldattention_b200.causal_dit import gated_residual, ln_modulate
    g = torch.Generator(device=dev()).manual_seed(0)
    make = lambda *shape: torch.randn(shape, generator=g, device=dev()).to(torch.bfloat16)
    b, f, n, c = 2, 3, 5, 256
    x, y, e = make(b, f * n, c), make(b, f * n, c), make(b, f, 6, c)
    for chunk in (e.chunk(6, dim=2), make(b, 2 * f, 6, c)[:, :f].chunk(6, dim=2)):     # frames of a longer tensor too
        scale, shift = chunk[1], chunk[2]
        want = ln_modulate(x, 1e-6, scale=scale, shift=shift, tokens_per_frame=n), gated_residual(x, y, scale, tokens_per_frame=n)
        scale, shift = scale.squeeze(2), shift.squeeze(2)
        assert torch.equal(ln_modulate(x, 1e-6, scale=scale, shift=shift, tokens_per_frame=n), want[0])
        assert torch.equal(gated_residual(x, y, scale, tokens_per_frame=n), want[1])
        strided = torch.stack([scale, shift], dim=-1)[..., 0]
        assert torch.equal(gated_residual(x, y, strided, tokens_per_frame=n), want[1])


def test_waiting_for_the_status_lets_other_threads_run():
    options = _inputs()
    want = _attend(**options, check_status=True)
    ticks, stop = [0], threading.Event()

    def tick():
        while not stop.wait(0.002):
            ticks[0] += 1

    torch.cuda.synchronize()
    thread = threading.Thread(target=tick)
    thread.start()
    try:
        torch.cuda._sleep(10 ** 9)          # about half a second of work in front of the call
        before, start = ticks[0], time.monotonic()
        got = _attend(**options, check_status=True)
        seen, waited = ticks[0] - before, time.monotonic() - start
    finally:
        stop.set()
        thread.join()
    assert waited > 0.2 and seen > 20 and torch.equal(got, want)


def _append_inputs(heads=2, seg=200, block=64, capacity=3):
    g = torch.Generator(device=dev()).manual_seed(0)
    slots = -(-seg // block)
    make = lambda n: torch.randn((1, n, heads, D), generator=g, device=dev()).to(torch.bfloat16)
    empty = lambda n: torch.zeros((1, n, heads, D), device=dev(), dtype=torch.bfloat16)
    proj = torch.randn((slots, seg), generator=g, device=dev()).to(torch.bfloat16)
    caches = [empty(capacity * seg), empty(capacity * seg), empty(capacity * slots), empty(capacity * slots)]
    return make(2 * seg), make(2 * seg), caches, dict(position=seg, segment_len=seg, k_proj_mat=proj, v_proj_mat=proj, block_size=block)


@pytest.mark.parametrize("which", [0, 1, 2, 3])
def test_append_into_caches_of_any_layout(which):
    from worldattention_b200.hsa.attention import append_kv
    k, v, caches, options = _append_inputs()
    append_kv(k, v, *caches, **options)
    _, _, others, _ = _append_inputs()
    others[which] = torch.zeros_like(others[which]).transpose(2, 3).contiguous().transpose(2, 3)       # channels are not side by side
    append_kv(k, v, *others, **options)
    for got, want in zip(others, caches):
        # the compressed slots may come from another kernel: one bf16 step of the largest value
        assert float((got.float() - want.float()).abs().max()) <= 2.0 ** -7 * float(want.float().abs().max())


@pytest.mark.parametrize("which", [1, 2, 3, 4, 5])
def test_append_needs_room_in_every_tensor(which):
    """v_new, the caches and the compressed tiers are addressed by the kernel: a row short of the need is an error on the host."""
    from worldattention_b200.hsa.attention import append_kv
    k, v, caches, options = _append_inputs()
    tensors = [k, v, *caches]
    append_kv(*tensors, **options)                        # two of three segments, up to the end
    before = [t.clone() for t in tensors]
    for short in (tensors[which][:, :-1], tensors[which][:, :, :1], tensors[which][..., :64], tensors[which][0]):
        with pytest.raises(ValueError):
            append_kv(*(short if i == which else t for i, t in enumerate(tensors)), **options)
    assert all(torch.equal(a, b) for a, b in zip(tensors, before))
    # a short last segment needs the slots of its own blocks only
    _, _, fresh, _ = _append_inputs()
    n = 200 + 70
    append_kv(k[:, :n], v[:, :n], *fresh[:2], *(t[:, :4 + 4 + 2] for t in fresh[2:]), **options)
    assert bool((fresh[2][:, 9] != 0).any()) and not bool((fresh[2][:, 10:] != 0).any())
