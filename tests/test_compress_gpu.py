"""compress_kv by the cluster kernel (float32 rows, or bf16 rows with a float32 projection) and by the tensor-core stream with items
of 64 and 128 columns, against float64 sums."""
import pytest
import torch

from tests.helpers import dev

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype,proj,heads,length,seg,block", [
    ("fp32", "fp32", 3, 700, 350, 64),       # two segments, rank 6
    ("fp32", "fp32", 1, 2048, 2048, 64),     # rank 32, the most that is accumulated in one pass
    ("fp32", "bf16", 2, 401, 200, 64),       # a last segment of one token
    ("bf16", "fp32", 12, 1170, 390, 64),
    ("bf16", "fp32", 4, 130, 65, 128),       # shorter than one share of a cluster
    ("bf16", "bf16", 12, 3 * 390, 390, 64),  # tensor-core stream: 72 items of 128 columns would leave SMs idle
    ("bf16", "bf16", 12, 9 * 200, 200, 128), # ... and 216 do not
    ("bf16", "bf16", 2, 1560, 1560, 64)])
def test_compress_kv(dtype, proj, heads, length, seg, block):
    import worldattention_b200 as wa
    g = torch.Generator(device=dev()).manual_seed(length)
    types = {"fp32": torch.float32, "bf16": torch.bfloat16}
    hsa = wa.hsa.HSAAttention(heads, 128, block_size=block, proj_segment_len=seg).to(dev())
    hsa.k_proj_mat.data = (torch.randn(hsa.k_proj_mat.shape, generator=g, device=dev()) * 0.1).to(types[proj])
    hsa.v_proj_mat.data = (torch.randn(hsa.v_proj_mat.shape, generator=g, device=dev()) * 0.1).to(types[proj])
    k, v = (torch.randn((2, length, heads, 128), generator=g, device=dev()).to(types[dtype]) for _ in range(2))
    got = hsa.compress_kv_cache(k, v)
    for out, x, e in zip(got, (k, v), (hsa.k_proj_mat, hsa.v_proj_mat)):
        want = []
        for start in range(0, length, seg):
            n = min(seg, length - start)
            r = min(e.shape[0], -(-n // block))
            want.append(torch.einsum("rt,bthd->brhd", e.detach()[:r, :n].double(), x[:, start:start + n].double()))
        want = torch.cat(want, dim=1)
        assert out.shape == want.shape and out.dtype == x.dtype
        # float32 sums of up to 2048 terms of size 0.1, and one rounding to the result's type
        step = 2.0 ** -8 if dtype == "bf16" else 0.0
        bound = want.abs() * step + 1e-5 * want.abs().max()
        assert bool(((out.double() - want).abs() <= bound).all())
