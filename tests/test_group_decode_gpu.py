"""Decoding attention of a group of heads over the rows they share, and 32-bit prompt attention, against float64: group sizes off the padded ones, row
widths at and off the lanes that read a row, splits as clusters and through the workspace, sequences of one key, every option."""
import math

import pytest
import torch

from tests.test_prompt_attention_gpu import DEV, F64, OPTIONS, nsq, reference  # noqa: F401  (nsq: the fixture)

pytestmark = pytest.mark.gpu
BF16, F32 = torch.bfloat16, torch.float32


def check(nsq, name, H, G, D, V, lens, pos0, dt, workspace, seed):
    g = torch.Generator(device=DEV).manual_seed(seed)
    T, B, cap = sum(lens), len(lens), (max(n + p for n, p in zip(lens, pos0)) + 127) // 128 * 128
    q = (torch.randn(T, H * D, generator=g, device=DEV) * 2).to(dt)
    k, v = torch.randn(B + 1, G, cap, D, generator=g, device=DEV).to(dt), torch.randn(B + 1, G, cap, V, generator=g, device=DEV).to(dt)
    slots = [B - b for b in range(B)]
    for b, (n, p) in enumerate(zip(lens, pos0)):
        k[slots[b], :, n + p:], v[slots[b], :, n + p:] = math.nan, math.nan
    o = OPTIONS[name](H, T, g)
    if "head_gate" in o:
        o["head_gate"] = o["head_gate"].to(dt)
    out = torch.empty(T, H * V, device=DEV, dtype=dt)
    opt = {a: x for a, x in o.items() if a not in ("r1", "r2", "sink")}
    if workspace:
        opt.update(workspace=nsq.attn_workspace(T, H, V, torch.device(DEV))[:None if workspace is True else workspace], max_keys=cap)
    nsq.attention(q, k, v, out, H, D ** -0.5, o.get("r1"), o.get("r2"), o.get("sink", False), nsq.Batch(slots, pos0, lens, torch.device(DEV)), **opt)
    off = 0
    for b, (n, p) in enumerate(zip(lens, pos0)):
        for h in range(H):
            kk, vv = k[slots[b], h * G // H, :n + p].to(F64), v[slots[b], h * G // H, :n + p].to(F64)
            want = reference(q[off:off + n, h * D:(h + 1) * D].to(F64), kk, vv, p, D ** -0.5, h, o) * o.get("out_scale", 1.0)
            if "head_gate" in o:
                want = want * torch.sigmoid(o["head_gate"][off:off + n, h].to(F64))[:, None]
            got = out[off:off + n, h * V:(h + 1) * V].to(F64)
            # 32-bit throughout: a score is a sum of D products (errors of 2^-24 each) of up to 2^4; a bfloat16 result is rounded at the end (2^-9 of it)
            bound = want.abs() * (2.0 ** -8 if dt == BF16 else 2.0 ** -20) + vv.abs().max() * 2.0 ** -16
            assert bool(((got - want).abs() <= bound).all()), (b, h, float(((got - want).abs() - bound).max()))
        off += n


DECODE = [  # heads, kv heads, dim, vdim, stored tokens of the sequences
    (4, 4, 128, 128, (0, 15, 16, 17, 1000)),
    (2, 1, 64, 64, (700,)),
    (6, 2, 72, 40, (2500, 31)),
    (16, 2, 192, 128, (130, 5)),
    (20, 1, 256, 256, (3000,)),                       # three blocks per group, the last of four heads; splits through the workspace
    (4, 1, 128, 64, tuple(range(100, 1700, 100))),    # sixteen tokens
]


@pytest.mark.parametrize("shape", DECODE)
@pytest.mark.parametrize("name", OPTIONS)
def test_group_decode(nsq, shape, name):  # noqa: F811
    H, G, D, V, pos0 = shape
    for dt in (BF16, F32):
        if dt == F32 and max(D, V) > 128:
            continue
        check(nsq, name, H, G, D, V, (1,) * len(pos0), pos0, dt, True, D + len(name))


def test_several_tokens_of_a_sequence(nsq):  # noqa: F811
    check(nsq, "bias", 8, 2, 128, 128, (3, 1, 5), (200, 0, 1000), BF16, True, 5)


def test_workspace_of_fewer_splits(nsq):  # noqa: F811
    """20 heads over 24 x 128 keys ask for 15 splits; a workspace that holds no more is enough, one float less is refused."""
    floats = 20 * 15 * (256 + 2)
    check(nsq, "plain", 20, 1, 256, 256, (1,), (3000,), BF16, floats, 3)
    with pytest.raises(nsq.NativeError, match="workspace too small"):
        check(nsq, "plain", 20, 1, 256, 256, (1,), (3000,), BF16, floats - 1, 3)


PROMPT32 = [
    (4, 2, 128, 128, (31, 32, 33, 65), (0, 63, 1, 64)),
    (3, 1, 68, 36, (130,), (0,)),
    (2, 2, 192, 64, (20, 1), (1900, 7)),    # a walk shared by a cluster
    (1, 1, 256, 128, (300,), (0,)),
]


@pytest.mark.parametrize("shape", PROMPT32)
@pytest.mark.parametrize("name", OPTIONS)
def test_prompt_attention_in_32_bits(nsq, shape, name):  # noqa: F811
    H, G, D, V, lens, pos0 = shape
    check(nsq, name, H, G, D, V, lens, pos0, F32, False, D + len(name))
