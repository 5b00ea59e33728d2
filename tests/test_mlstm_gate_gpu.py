"""The output gate of the matrix-memory recurrence in every form, down to gates whose sigmoid is below the smallest normal number."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV, BF16, F64 = torch.device("cuda:0"), torch.bfloat16, torch.float64


@pytest.mark.parametrize("n,V", [(300, 128), (300, 40), (100, 128), (500, 512), (1, 64)])   # side by side, one chunk after the other, token by token
def test_closed_gates(n, V):
    from promptcache_b200 import _native_seq as nsq
    g = torch.Generator().manual_seed(V)
    H, D = 1, 64
    proj, offs = torch.randn(n, 2 * H * D + 2 * H * V, generator=g).to(BF16), (0, H * D, 2 * H * D, 2 * H * D + H * V)
    ig, fg = torch.randn(n, H, generator=g), torch.nn.functional.logsigmoid(torch.randn(n, H, generator=g) + 3)
    outs = []
    for z in (0.0, -6.0, -86.0, -88.0):
        p = proj.clone()
        p[:, offs[3]:] = z
        s, nn, m = torch.zeros(1, H, D, V, device=DEV), torch.zeros(1, H, D, device=DEV), torch.zeros(1, H, device=DEV)
        out = torch.empty(n, H * V, device=DEV, dtype=BF16)
        nsq.mlstm_scan(p.to(DEV), offs, ig.to(DEV), fg.to(DEV), torch.full((H * V,), 64.0, dtype=BF16, device=DEV), out, s, nn, m, 1e-5, nsq.Batch([0], [0], [n], DEV))
        outs.append((z, out.cpu().to(F64)))
    open_ = outs[0][1] * 2          # sigmoid(0) = 1/2
    for z, out in outs[1:]:
        want = open_ * torch.sigmoid(torch.tensor(z, dtype=F64))
        # two results rounded to bfloat16 (2^-9 each; below 2^-126 its numbers are 2^-133 apart), a sigmoid that is a 32-bit number (2^-149 apart down there, times 64 and
        # the normed result)
        assert float(((out - want).abs() - want.abs() * 2.0 ** -7).max()) <= 2.0 ** -133 + 2.0 ** -149 * 512, z
