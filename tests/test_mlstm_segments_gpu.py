"""The matrix-memory recurrence where few heads walk over many chunks (the walk is cut into segments side by side), and with gates and results that do not start
on 16 bytes, against the float64 recurrence."""
import pytest
import torch

from tests import mutolix_oracle as O

pytestmark = pytest.mark.gpu
DEV, BF16, F64 = torch.device("cuda:0"), torch.bfloat16, torch.float64


@pytest.mark.parametrize("H,D,V,gap,steps", [
    (1, 64, 128, 0, [(1200, 200), (300, 1301)]),     # six segments of which the short entry fills four; a continued state at the start of the first
    (2, 80, 72, 2, [(961,), (1100,)]),               # tiles that reach past rows and columns; gates on 4 bytes
    (1, 256, 512, 2, [(449,)]),
    (1, 128, 256, 2, [(200,)]),
    (2, 64, 128, 0, [(577, 129, 65), (64, 641, 1)]),  # five segments of two chunks: entries that fill the first, or part of it
    (4, 128, 128, 0, [(705, 400)]),                  # as many segments as there are SMs for
])
def test_long_walks_of_few_heads(H, D, V, gap, steps):
    from promptcache_b200 import _native_seq as nsq
    g = torch.Generator().manual_seed(D + V)
    B = len(steps[0])
    s, n, m = torch.full((B, H, D, V), 9.0, device=DEV), torch.full((B, H, D), 9.0, device=DEV), torch.full((B, H), 9.0, device=DEV)
    w = (1 + 0.1 * torch.randn(H * V, generator=g)).to(BF16)
    states, pos = [None] * B, [0] * B
    offs = (0, H * D, 2 * H * D, 2 * H * D + H * V + gap)
    for lens in steps:
        T = sum(lens)
        proj = torch.randn(T, 2 * H * D + 2 * H * V + 8, generator=g).to(BF16)
        ig, fg = torch.randn(T, H, generator=g) * 2, torch.nn.functional.logsigmoid(torch.randn(T, H, generator=g) * 2 + 3)
        out = torch.empty(T * H * V + gap, device=DEV, dtype=BF16)[gap:].view(T, H * V)
        nsq.mlstm_scan(proj.to(DEV), offs, ig.to(DEV), fg.to(DEV), w.to(DEV), out, s, n, m, 1e-5, nsq.Batch(range(B), pos, lens, DEV))
        o = 0
        for b, ln in enumerate(lens):
            x = proj[o:o + ln].to(F64)
            q, k, v = x[:, :offs[1]].view(ln, H, D) * D ** -0.5, x[:, offs[1]:offs[2]].view(ln, H, D), x[:, offs[2]:offs[2] + H * V].view(ln, H, V)
            want, states[b] = O.mlstm_recurrence(q, k, v, ig[o:o + ln].to(F64), fg[o:o + ln].to(F64), states[b])
            want = O.rms(want, 1e-5).reshape(ln, H * V) * w.to(F64) * torch.sigmoid(x[:, offs[3]:offs[3] + H * V])
            got = out[o:o + ln].cpu().to(F64)
            # rounded to bfloat16 (2^-9); weights and state keep 16 bits of what they add up to
            assert float(((got - want).abs() - want.abs() * 2.0 ** -8).max()) <= 2.0 ** -12 * float(want.abs().max()), b
            for have, ref in zip((s, n, m), states[b]):
                have = have[b].cpu().to(F64)
                assert float((have - ref).abs().max()) <= 3e-5 * float(ref.abs().max()) + 1e-6
            pos[b] += ln
            o += ln


@pytest.mark.parametrize("H,D,V,lens", [(4, 128, 128, (500, 64, 1)), (16, 128, 256, (1601,)), (2, 80, 64, (449,))])
def test_normaliser_token_by_token(H, D, V, lens):
    """Walks in one piece add the normaliser's terms in the order of the tokens within a chunk and of the chunks, whichever warps do: with gates that weigh every token by 1 the sums can be
    formed here, bit for bit."""
    from promptcache_b200 import _native_seq as nsq
    g = torch.Generator().manual_seed(D)
    B, T = len(lens), sum(lens)
    proj, ones = torch.randn(T, 2 * H * D + 2 * H * V, generator=g).to(BF16), torch.ones(H * V, dtype=BF16, device=DEV)
    s, n, m = torch.zeros(B, H, D, V, device=DEV), torch.zeros(B, H, D, device=DEV), torch.zeros(B, H, device=DEV)
    nsq.mlstm_scan(proj.to(DEV), (0, H * D, 2 * H * D, 2 * H * D + H * V), torch.zeros(T, H, device=DEV), torch.zeros(T, H, device=DEV), ones, torch.empty(T, H * V, dtype=BF16, device=DEV),
                   s, n, m, 1e-5, nsq.Batch(range(B), [0] * B, lens, DEV))
    k, o = proj[:, H * D:2 * H * D].float(), 0
    for b, ln in enumerate(lens):
        want = torch.zeros(H * D)
        for c in range(0, ln, 64):
            own = torch.zeros(H * D)
            for t in range(c, min(c + 64, ln)):
                own = own + k[o + t]
            want = want + own
        assert torch.equal(n[b].cpu().flatten(), want), b
        o += ln
