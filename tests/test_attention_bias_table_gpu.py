"""A tabulated bias that hides keys (minus infinity), in the attention over the slot pool: whole tiles of a walk may be hidden before the first visible key."""
import math

import pytest
import torch

from tests.test_prompt_attention_gpu import DEV, F64, nsq, reference  # noqa: F401  (nsq: the fixture)

pytestmark = pytest.mark.gpu
BF16, F32 = torch.bfloat16, torch.float32


def bound(want, v, dt):
    """As in the tests of finite inputs: 32-bit sums, in bfloat16 weights of 16 bits and a rounded result."""
    return want.abs() * (2.0 ** -8 if dt == BF16 else 2.0 ** -19) + v.abs().max() * (2.0 ** -13 if dt == BF16 else 2.0 ** -16)


@pytest.mark.parametrize("dt", [BF16, F32])
@pytest.mark.parametrize("H,G,D,V,stored,lens", [
    (4, 1, 128, 128, (99, 700, 64, 3), 1),       # decoding, clusters
    (6, 2, 64, 64, (2500,), 1),
    (20, 1, 256, 256, (3000,), 1),               # splits through the workspace
    (2, 1, 128, 64, (300, 0), 40),               # prompts
])
def test_bias_table_that_hides_distant_keys(nsq, dt, H, G, D, V, stored, lens):  # noqa: F811
    if dt == F32 and max(D, V) > 128:
        pytest.skip("wider than the 32-bit kernels' rows")
    g = torch.Generator(device=DEV).manual_seed(D + H)
    B, T, cap = len(stored), len(stored) * lens, (max(stored) + lens + 127) // 128 * 128
    q = (torch.randn(T, H * D, generator=g, device=DEV) * 2).to(dt)
    k, v = torch.randn(B, G, cap, D, generator=g, device=DEV).to(dt), torch.randn(B, G, cap, V, generator=g, device=DEV).to(dt)
    table = torch.randn(H, 66, generator=g, device=DEV)
    table[:, 65] = -math.inf                     # every distance of 65 and more
    out = torch.full((T, H * V), 7.0, device=DEV, dtype=dt)
    nsq.attention(q, k, v, out, H, D ** -0.5, None, None, False, nsq.Batch(range(B), stored, [lens] * B, torch.device(DEV)), bias_table=table,
                  workspace=nsq.attn_workspace(T, H, V, torch.device(DEV)), max_keys=cap)
    for b, p in enumerate(stored):
        for h in range(H):
            kk, vv = k[b, h * G // H, :p + lens].to(F64), v[b, h * G // H, :p + lens].to(F64)
            rows = slice(b * lens, (b + 1) * lens)
            want = reference(q[rows, h * D:(h + 1) * D].to(F64), kk, vv, p, D ** -0.5, h, dict(bias_table=table))
            got = out[rows, h * V:(h + 1) * V].to(F64)
            assert bool(((got - want).abs() <= bound(want, vv, dt)).all()), (b, h)
