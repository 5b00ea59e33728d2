"""The read-out of gated linear attention in bfloat16 prompts keeps all 24 bits of its 32-bit operands: results that are what is left of large products."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV, BF16, F64 = torch.device("cuda:0"), torch.bfloat16, torch.float64


@pytest.mark.parametrize("H,D,V,n", [(2, 64, 72, 64), (1, 256, 512, 100), (3, 16, 8, 33), (1, 128, 256, 129)])
def test_results_left_of_cancelling_products(H, D, V, n):
    from promptcache_b200 import _native_seq as nsq
    g = torch.Generator().manual_seed(D)
    offs, eps = (0, H * D, 2 * H * D, 2 * H * D + H * V), 0.0
    # neighbouring channels of the state share a large part, neighbouring channels of q have opposite signs: what is left is 2^-10 of the products
    s = torch.randn(1, H, D // 2, V, generator=g).repeat_interleave(2, 2) + torch.randn(1, H, D, V, generator=g) * 2.0 ** -10
    x = torch.randn(n, H, D // 2, generator=g)
    proj = torch.zeros(n, 2 * H * D + 2 * H * V)
    proj[:, :H * D] = torch.stack([x, -x], -1).reshape(n, H * D)
    proj[:, H * D:2 * H * D] = torch.randn(n, H * D, generator=g) * 2.0 ** -12
    proj[:, 2 * H * D:] = torch.randn(n, 2 * H * V, generator=g)
    proj = proj.to(BF16)
    w, ld, out = torch.ones(V, dtype=BF16), torch.zeros(n, H * D), torch.empty(n, H * V, device=DEV, dtype=BF16)
    nsq.gla_scan(proj.to(DEV), offs, ld.to(DEV), w.to(DEV), out, s.to(DEV), eps, nsq.Batch([0], [5], [n], DEV))
    p, S, res = proj.to(F64), s[0].to(F64), torch.empty(n, H, V, dtype=F64)
    for t in range(n):
        S = S + p[t, H * D:2 * H * D].view(H, D, 1) * p[t, offs[2]:offs[3]].view(H, 1, V)
        res[t] = torch.einsum("hd,hdv->hv", p[t, :H * D].view(H, D) * D ** -0.5, S)
    gate = p[:, offs[3]:]
    want = (res / torch.sqrt((res * res).mean(-1, keepdim=True))).reshape(n, H * V) * gate * torch.sigmoid(gate)
    got = out.cpu().to(F64)
    # a result is rounded to bfloat16 (2^-9); sums of products that are 2^10 times as large, in 32 bits: 2^-24 * 2^10 times a few, of a normed result of
    # up to 4.  (16 bits of the operands: 2^-17 * 2^10 of it.)
    assert float(((got - want).abs() - want.abs() * 2.0 ** -8).max()) <= 2.0 ** -11 * 4
