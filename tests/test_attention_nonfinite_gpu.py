"""K / V rows that hold NaN or infinity, in the prompt attention over the slot pool: a query's result depends on the keys it sees and on nothing else,
whatever stands in the others."""
import math

import pytest
import torch

from tests.test_attention_bias_table_gpu import BF16, DEV, F32, F64, bound, nsq, reference  # noqa: F401  (nsq: the fixture)

pytestmark = pytest.mark.gpu
OPTS = {"plain": {}, "window": dict(softcap=20.0, window=70, keep_first=5), "chunk": dict(chunk=96), "cap": dict(softcap=30.0)}


@pytest.mark.parametrize("dt", [BF16, F32])
@pytest.mark.parametrize("name", OPTS)
@pytest.mark.parametrize("bad", [(201, "k", math.nan), (202, "v", math.nan), (127, "v", math.inf), (200, "kv", math.nan)])
@pytest.mark.parametrize("H,stored,new", [(1, 0, 300), (2, 100, 200), (1, 0, 2049), (40, 0, 600)])   # (clusters of several sizes; a launch of many tiles)
def test_rows_that_are_not_finite_reach_only_queries_that_see_them(nsq, dt, name, bad, H, stored, new):  # noqa: F811
    key, where, value = bad
    D = V = 128
    g = torch.Generator(device=DEV).manual_seed(key + H)
    q = (torch.randn(new, H * D, generator=g, device=DEV) * 2).to(dt)
    cap, n = (stored + new + 127) // 128 * 128, stored + new
    k, v = torch.randn(1, H, cap, D, generator=g, device=DEV).to(dt), torch.randn(1, H, cap, V, generator=g, device=DEV).to(dt)
    kc, vc = k.to(F64), v.to(F64)
    if "k" in where:
        k[0, :, key, 3] = value
    if "v" in where:
        v[0, :, key] = value
    out = torch.full((new, H * V), 7.0, device=DEV, dtype=dt)
    o = OPTS[name]
    nsq.attention(q, k, v, out, H, D ** -0.5, None, None, False, nsq.Batch([0], [stored], [new], torch.device(DEV)), **o)
    i = torch.arange(stored, n, device=DEV)
    sees = i >= key
    if "window" in o:
        sees &= i - key < o["window"]
    if "chunk" in o:
        sees &= i // o["chunk"] == key // o["chunk"]
    for h in range(0, H, 7):
        want = reference(q[:, h * D:(h + 1) * D].to(F64), kc[0, h, :n], vc[0, h, :n], stored, D ** -0.5, h, o)
        got = out[:, h * V:(h + 1) * V].to(F64)
        err = (got - want).abs() - bound(want, vc[0, h, :n], dt)
        assert bool((err[~sees] <= 0).all()), (h, float(err[~sees].max()))
        assert not bool(got[sees].isfinite().any())
