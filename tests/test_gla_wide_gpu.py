"""Gated linear attention of prompts over heads of more than 256 channels, at and beyond the widest that a chunk's preparation holds."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV, F64 = torch.device("cuda:0"), torch.float64


@pytest.mark.parametrize("dt", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("D", [260, 288, 289, 291, 292, 293, 296])
def test_wide_heads(dt, D):
    from promptcache_b200 import _native_seq as nsq
    H, V, n, eps = 1, 24, 100, 1e-5
    g = torch.Generator().manual_seed(D)
    offs = (0, H * D, 2 * H * D, 2 * H * D + H * V)
    proj = torch.randn(n, 2 * H * D + 2 * H * V, generator=g).to(dt)
    ld = torch.nn.functional.logsigmoid(torch.randn(n, H * D, generator=g)) / 4
    w = (1 + 0.1 * torch.randn(V, generator=g)).to(dt)
    s, out = torch.zeros(1, H, D, V, device=DEV), torch.empty(n, H * V, device=DEV, dtype=dt)
    nsq.gla_scan(proj.to(DEV), offs, ld.to(DEV), w.to(DEV), out, s, eps, nsq.Batch([0], [0], [n], DEV))
    x, S, res = proj.to(F64), torch.zeros(D, V, dtype=F64), torch.empty(n, V, dtype=F64)
    for t in range(n):
        S = S * torch.exp(ld[t].to(F64))[:, None] + x[t, D:2 * D, None] * x[t, None, offs[2]:offs[3]]
        res[t] = (x[t, :D] * D ** -0.5) @ S
    gate = x[:, offs[3]:]
    want = res / torch.sqrt((res * res).mean(-1, keepdim=True) + eps) * w.to(F64) * gate * torch.sigmoid(gate)
    # the result is rounded to its type; 32-bit sums of ~ 2^9 terms whose decays are exponentials of differences of sums of up to 2^6
    rel = 2.0 ** -8 if dt == torch.bfloat16 else 2.0 ** -16
    assert float(((out.cpu().to(F64) - want).abs() - want.abs() * rel).max()) <= 2.0 ** -14 * float(want.abs().max())
    assert float((s[0, 0].cpu().to(F64) - S).abs().max()) <= 2.0 ** -17 * float(S.abs().max())
