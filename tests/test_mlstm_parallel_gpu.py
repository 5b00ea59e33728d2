"""The matrix-memory recurrence with its chunks side by side against the float64 recurrence: chunk edges, every padded width of the read-out, state rows off a
multiple of 32, unequal entries, continued states, and the state handed on."""
import pytest
import torch

from tests import mutolix_oracle as O

pytestmark = pytest.mark.gpu
DEV, BF16, F32, F64 = torch.device("cuda:0"), torch.bfloat16, torch.float32, torch.float64


@pytest.fixture(scope="module")
def nsq():
    from promptcache_b200 import _native_seq
    _native_seq.load()
    return _native_seq


@pytest.mark.parametrize("H,D,V,steps", [
    (2, 48, 40, [(193, 256, 1)]),                 # 128 columns padded, rows off 32, an entry of one token
    (1, 128, 200, [(257, 30), (320, 64)]),        # 256 padded, a second step that continues both
    (1, 16, 504, [(450,)]),                       # 512 padded
    (2, 256, 128, [(200,), (63,), (448,)]),       # side by side, one after the other, side by side
])
def test_chunks_side_by_side(nsq, H, D, V, steps):
    g = torch.Generator().manual_seed(D + V)
    B = len(steps[0])
    s, n, m = torch.full((B, H, D, V), 9.0, device=DEV), torch.full((B, H, D), 9.0, device=DEV), torch.full((B, H), 9.0, device=DEV)
    w = (1 + 0.1 * torch.randn(H * V, generator=g)).to(BF16)
    states, pos = [None] * B, [0] * B
    offs = (0, H * D, 2 * H * D, 2 * H * D + H * V)
    for lens in steps:
        T = sum(lens)
        proj = torch.randn(T, 2 * H * D + 2 * H * V, generator=g).to(BF16)
        ig, fg = torch.randn(T, H, generator=g) * 2, torch.nn.functional.logsigmoid(torch.randn(T, H, generator=g) * 2 + 2)
        out = torch.empty(T, H * V, device=DEV, dtype=BF16)
        slots = [B - 1 - b for b in range(B)]
        nsq.mlstm_scan(proj.to(DEV), offs, ig.to(DEV), fg.to(DEV), w.to(DEV), out, s, n, m, 1e-5, nsq.Batch(slots, pos, lens, DEV))
        o = 0
        for b, ln in enumerate(lens):
            x = proj[o:o + ln].to(F64)
            q, k, v, gate = x[:, :offs[1]].view(ln, H, D) * D ** -0.5, x[:, offs[1]:offs[2]].view(ln, H, D), x[:, offs[2]:offs[3]].view(ln, H, V), x[:, offs[3]:]
            want, states[b] = O.mlstm_recurrence(q, k, v, ig[o:o + ln].to(F64), fg[o:o + ln].to(F64), states[b])
            want = O.rms(want, 1e-5).reshape(ln, H * V) * w.to(F64) * torch.sigmoid(gate)
            got = out[o:o + ln].cpu().to(F64)
            # rounded to bfloat16 (2^-9); weights and state keep 16 bits of what they add up to
            assert float(((got - want).abs() - want.abs() * 2.0 ** -8).max()) <= 2.0 ** -12 * float(want.abs().max()), b
            for have, ref in zip((s, n, m), states[b]):
                have = have[slots[b]].cpu().to(F64)
                assert float((have - ref).abs().max()) <= 3e-5 * float(ref.abs().max()) + 1e-6
            pos[b] += ln
            o += ln
