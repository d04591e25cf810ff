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


def test_a_streams_workspace_grows_and_is_kept():
    sizes = [(70, 130), (700, 6000), (130, 200), (1500, 9000), (70, 130)]
    options = [_inputs(lq, lkv, seed=i) for i, (lq, lkv) in enumerate(sizes)]
    want = []
    for o in options:                                   # a stream of its own each
        stream = torch.cuda.Stream()
        stream.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(stream):
            want.append(_attend(**o))
        torch.cuda.current_stream().wait_stream(stream)
    got = [_attend(**o) for o in options]               # one after the other on one stream, nothing waits
    assert all(torch.equal(a, b) for a, b in zip(got, want))


def test_workspaces_of_many_streams_are_bounded():
    options = _inputs()
    want = _attend(**options)
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream() for _ in range(64)]
    streams = list({s.cuda_stream: s for s in streams}.values())          # the pool hands streams out again
    extra = [torch.cuda.ExternalStream(_new_stream()) for _ in range(48)]
    before, outs = torch.cuda.memory_allocated(), []
    for stream in streams + extra:
        with torch.cuda.stream(stream):
            outs.append(_attend(**options))
    torch.cuda.synchronize()
    assert len(streams) + len(extra) >= 48 and all(torch.equal(o, want) for o in outs)
    results = sum(o.untyped_storage().nbytes() for o in outs)
    assert torch.cuda.memory_allocated() - before <= 32 * (1 << 20) + results + len(outs) * 512       # 32 of the least size


def _new_stream():
    """A CUDA stream outside the framework's pool, never destroyed."""
    import ctypes
    rt = ctypes.CDLL("libcudart.so.12")
    handle = ctypes.c_void_p()
    assert rt.cudaStreamCreateWithFlags(ctypes.byref(handle), 1) == 0
    return handle.value


def test_a_captured_call_keeps_its_workspace_to_itself():
    small, large = _inputs(130, 200, seed=1), _inputs(700, 6000, seed=2)
    want = _attend(**small), _attend(**large)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        got = _attend(**small), _attend(**large)
    for _ in range(2):
        for o in got:
            o.zero_()
        graph.replay()
        eager = [_attend(**_inputs(900, 7000, seed=3)) for _ in range(3)]          # grows and uses the kept one behind the replay
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1]) and torch.equal(eager[0], eager[2])


@pytest.mark.parametrize("generic", [False, True])
def test_partials_of_a_shard_use_the_same_workspace(generic):
    from worldattention_b200.hsa.branches import hsa_partials, hsa_partials_packed, merge_partials, record_floats
    options = _inputs(130, 512, block=64)
    kc, vc = options["k"][:, ::64].contiguous(), options["v"][:, ::64].contiguous()
    out, (index, num, _, _) = _attend(**options, k_coarse=kc, v_coarse=vc, return_routing=True)
    torch.cuda.synchronize()
    before = torch.cuda.memory_allocated()
    shard = (options["q"], options["k"], options["v"], kc, vc, index, num, 64)
    sparse, lse, linear, _, used = hsa_partials(*shard, force_generic=generic)
    assert used is not generic
    want = sparse + torch.sigmoid(options["q"].float()) * linear              # a call without gate weights
    assert float((out.float() - want).abs().max()) <= 2.0 ** -6 * float(want.abs().max())
    records = torch.zeros((1, 130, 2, record_floats(D)), device=dev())
    assert hsa_partials_packed(*shard, records)
    assert float((records[..., :D] - sparse).abs().max()) <= 2.0 ** -6 * float(sparse.abs().max())
    del sparse, lse, linear, records, want
    assert torch.cuda.memory_allocated() - before <= 1 << 16          # no second workspace
    wide = torch.zeros((1, 130, 2, 64), device=dev(), dtype=torch.bfloat16)
    assert not hsa_partials_packed(wide, wide, wide, wide, wide, index[..., :3].contiguous(), num, 64,
                                   torch.zeros((1, 130, 2, record_floats(64)), device=dev()))
