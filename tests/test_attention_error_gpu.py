"""The error of the bf16 layer against float64: no more than that of the roundings it is documented to have (probabilities, the sparse
branch, the gate and the result to bf16), each made here in float64 arithmetic on the same selection."""
import math

import pytest
import torch

from tests.helpers import dev

pytestmark = pytest.mark.gpu
D = 128


def _softmax(s, v, rounded):
    p = torch.exp(s - s.amax(-1, keepdim=True))
    if rounded:      # against any reference point: only where it is the row's maximum is the largest probability exactly one
        p = p * (1 + torch.rand(p.shape[0], 1, device=p.device, dtype=p.dtype, generator=torch.Generator(p.device).manual_seed(0)))
    total = p.sum(-1, keepdim=True)
    return (p.to(torch.bfloat16).double() if rounded else p) @ v / total


def _layer(q, k, v, kc, vc, lin, index, num, block, rounded):
    step = (lambda t: t.to(torch.bfloat16).double()) if rounded else (lambda t: t)
    q, k, v, kc, vc, w, b = (t.double() for t in (q, k, v, kc, vc, lin.weight, lin.bias))
    if rounded:
        w = step(w)                           # an operand of a matrix product
    out = torch.empty_like(q)
    for h in range(q.shape[2]):
        s = q[0, :, h] @ k[0, :, h].T / math.sqrt(D)
        for i in range(num.shape[2]):
            rows = slice(i * block, (i + 1) * block)
            chosen = torch.zeros(-(-k.shape[1] // block), dtype=torch.bool, device=q.device)
            chosen[index[0, h, i, : int(num[0, h, i])].long()] = True
            keys = chosen.repeat_interleave(block)[: k.shape[1]]
            out[0, rows, h] = step(_softmax(s[rows][:, keys], v[0, keys, h], rounded))
        gate = step(torch.sigmoid(q[0, :, h] @ w.T + b))
        out[0, :, h] += gate * _softmax(q[0, :, h] @ kc[0, :, h].T / math.sqrt(D), vc[0, :, h], rounded)
    return step(out)


# 128-token blocks; 64-token blocks in pairs and alone; `scale` times the usual queries and keys (rows outgrow their reference points)
@pytest.mark.parametrize("block,heads,q_len,kv_len,scale", [(128, 12, 1990, 4990, 1), (64, 12, 1990, 4990, 1), (64, 12, 390, 1170, 1),
                                                            (128, 12, 1990, 4990, 3), (64, 12, 1990, 4990, 3)])
def test_error_is_that_of_the_documented_roundings(block, heads, q_len, kv_len, scale):
    from worldattention_b200.hsa import hsa_attention
    g = torch.Generator(device=dev()).manual_seed(block + q_len)
    draw = lambda n: torch.randn(1, n, heads, D, generator=g, device=dev())
    patch = lambda n: torch.randn(1, -(-n // 130), heads, D, generator=g, device=dev()).repeat_interleave(130, 1)[:, :n]
    q, k, v = ((draw(q_len) + patch(q_len)) * scale, (draw(kv_len) + patch(kv_len)) * scale, draw(kv_len))
    kc, vc = draw(200) * 0.5 * scale, draw(200) * 0.5
    q, k, v, kc, vc = (t.bfloat16() for t in (q, k, v, kc, vc))
    lin = torch.nn.Linear(D, D).to(dev())
    with torch.no_grad():
        lin.weight.copy_(torch.randn(D, D, generator=g, device=dev()) * 0.05)
        lin.bias.copy_(torch.randn(D, generator=g, device=dev()) * 0.2)
        out, (index, num, _, used) = hsa_attention(q, k, v, k_coarse=kc, v_coarse=vc, k_proj_mat=None, v_proj_mat=None, gate_lin=lin,
                                                   block_size=block, return_routing=True, check_status=True)
        exact, rounded = (_layer(q, k, v, kc, vc, lin, index, num, block, r) for r in (False, True))
    assert used
    error = lambda x: float((x.double() - exact).norm() / exact.norm())
    got, documented = error(out), error(rounded)
    # beside these: the exponential of every eighth pair of columns (2.1e-4 in the mean square), the sums in float32 and a sigmoid
    # from tanh.approx (2^-11 of the gate at most), independent of the roundings: added in squares
    assert got <= math.hypot(documented, 3e-4) * 1.01, (got, documented)
