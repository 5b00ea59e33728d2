"""Prompt attention against float64 at sizes where a walk over the keys is not shared by a cluster, or by two blocks: several rounds of blocks per SM, the last of
them short and in reversed order (32-bit tiles), tiles from both ends of a sequence or neighbours without a merge (tcgen05).  The output starts as NaN, so a
tile that no block takes shows."""
import math

import pytest
import torch

from tests.test_attention_bias_table_gpu import BF16, DEV, F32, F64, bound, nsq, reference  # noqa: F401  (nsq: the fixture)
from tests.test_prompt_attention_gpu import OPTIONS

pytestmark = pytest.mark.gpu


def compare(nsq, name, dt, H, G, D, V, lens, pos0):  # noqa: F811
    g = torch.Generator(device=DEV).manual_seed(H + D)
    T, B, cap = sum(lens), len(lens), (max(n + p for n, p in zip(lens, pos0)) + 127) // 128 * 128
    q = (torch.randn(T, H * D, generator=g, device=DEV) * 2).to(dt)
    k, v = torch.randn(B, G, cap, D, generator=g, device=DEV).to(dt), torch.randn(B, G, cap, V, generator=g, device=DEV).to(dt)
    o = OPTIONS[name](H, T, g)
    out = torch.full((T, H * V), math.nan, device=DEV, dtype=dt)
    opt = {a: x for a, x in o.items() if a not in ("r1", "r2", "sink")}
    nsq.attention(q, k, v, out, H, D ** -0.5, o.get("r1"), o.get("r2"), o.get("sink", False), nsq.Batch(range(B), pos0, lens, torch.device(DEV)), **opt)
    off = 0
    for b, (n, p) in enumerate(zip(lens, pos0)):
        for h in range(H):
            kk, vv = k[b, h * G // H, :n + p].to(F64), v[b, h * G // H, :n + p].to(F64)
            want = reference(q[off:off + n, h * D:(h + 1) * D].to(F64), kk, vv, p, D ** -0.5, h, o) * o.get("out_scale", 1.0)
            got = out[off:off + n, h * V:(h + 1) * V].to(F64)
            assert bool(((got - want).abs() <= bound(want, vv, dt)).all()), (b, h)
        off += n


@pytest.mark.parametrize("dt,H,G,D,V,lens,pos0", [
    (F32, 8, 2, 64, 36, (2049,), (0,)),             # 520 blocks: three rounds of 148 and a short one, reversed
    (F32, 8, 2, 128, 128, (1024,), (0,)),           # two blocks per walk
    (F32, 16, 4, 64, 64, (300, 33, 1, 700), (0, 100, 5, 31)),
    (BF16, 14, 7, 128, 128, (2049,), (0,)),         # tiles from both ends, an odd number of them
    (BF16, 16, 4, 64, 128, (2311, 130), (0, 64)),   # more than one round of blocks
    (BF16, 40, 8, 128, 64, (600,), (0,)),           # neighbours
    (BF16, 8, 2, 192, 128, (900, 17, 300), (0, 1000, 63)),
])
@pytest.mark.parametrize("name", ["plain", "bias", "window", "chunk"])
def test_forms(nsq, dt, H, G, D, V, lens, pos0, name):  # noqa: F811
    compare(nsq, name, dt, H, G, D, V, lens, pos0)
