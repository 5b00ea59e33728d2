"""Gated linear attention of bfloat16 prompts against float64: chunk remainders, channels and columns at and off the tensor-core tiles, unequal entries, a
continued state."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV, BF16, F64 = torch.device("cuda:0"), torch.bfloat16, torch.float64


@pytest.mark.parametrize("H,D,V", [(2, 16, 8), (1, 48, 136), (3, 20, 12), (1, 256, 512), (2, 64, 520)])
def test_chunks(H, D, V):
    from promptcache_b200 import _native_seq as nsq
    g = torch.Generator().manual_seed(D + V)
    offs, eps = (0, H * D, 2 * H * D, 2 * H * D + H * V), 1e-5
    s = torch.full((2, H, D, V), 9.0, device=DEV)
    w = (1 + 0.1 * torch.randn(V, generator=g)).to(BF16)
    states, pos = [torch.zeros(H, D, V, dtype=F64) for _ in range(2)], [0, 0]
    for lens in ((65, 127), (64, 33)):
        T = sum(lens)
        proj = torch.randn(T, 2 * H * D + 2 * H * V, generator=g).to(BF16)
        ld = torch.nn.functional.logsigmoid(torch.randn(T, H * D, generator=g)) / 4
        ld[5, :H * D // 2] = -40.0    # half of the channels forget everything
        out = torch.empty(T, H * V, device=DEV, dtype=BF16)
        nsq.gla_scan(proj.to(DEV), offs, ld.to(DEV), w.to(DEV), out, s, eps, nsq.Batch([1, 0], pos, lens, DEV))
        o = 0
        for b, n in enumerate(lens):
            x = proj[o:o + n].to(F64)
            q, k, v = x[:, :offs[1]].view(n, H, D) * D ** -0.5, x[:, offs[1]:offs[2]].view(n, H, D), x[:, offs[2]:offs[3]].view(n, H, V)
            dec, res = torch.exp(ld[o:o + n].to(F64)).view(n, H, D, 1), torch.empty(n, H, V, dtype=F64)
            for t in range(n):
                states[b] = states[b] * dec[t] + k[t][..., None] * v[t][:, None, :]
                res[t] = torch.einsum("hdv,hd->hv", states[b], q[t])
            gate = x[:, offs[3]:]
            want = (res / torch.sqrt((res * res).mean(-1, keepdim=True) + eps) * w.to(F64)).reshape(n, H * V) * gate * torch.sigmoid(gate)
            got = out[o:o + n].cpu().to(F64)
            # rounded to bfloat16 (2^-9); the read-out's operands keep 16 bits, a norm over few small results enlarges that
            assert float(((got - want).abs() - want.abs() * 2.0 ** -8).max()) <= 2.0 ** -11 * float(want.abs().max())
            have = s[1 - b].cpu().to(F64)
            # a 32-bit state whose decays are exponentials of differences of running sums of up to 2^6: 2^-24 * 2^6 of each sum
            assert float((have - states[b]).abs().max()) <= 2 * 2.0 ** -18 * float(states[b].abs().max())
            pos[b] += n
            o += n
