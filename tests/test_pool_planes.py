"""Prompt attention through tensor maps: the maps end where the pool ends, and dense K/V of a step whose rows the maps' boxes do not divide are read without them."""
import ctypes

import pytest
import torch

from tests.test_prompt_attention_route import wanted

DEV, BF16, F64 = "cuda:0", torch.bfloat16, torch.float64


def test_dense_rows_off_the_boxes_ask_for_no_scratch():
    from promptcache_b200 import _native_seq as nsq
    for d, v, yes in ((128, 128, True), (192, 128, True), (96, 128, False), (128, 72, False), (136, 80, False)):
        assert wanted(16, 4, d, v, (300,), (0,), impl=4)
        assert wanted(16, 4, d, v, (300,), (0,), impl=4, pool_slot=1 << 20) is yes, (d, v)
    assert ctypes.sizeof(nsq.pcs_attn_params) == 280


@pytest.mark.gpu
@pytest.mark.parametrize("H,G,D,V,n,impl", [(4, 2, 128, 128, 300, 0), (2, 2, 64, 64, 200, 0), (4, 2, 128, 128, 300, 4), (4, 2, 192, 128, 140, 4)])
def test_maps_end_where_the_pool_ends(H, G, D, V, n, impl):
    """A slot behind the pool's last one, in memory that is there: its rows are not read."""
    from promptcache_b200 import _native_seq as nsq
    q = torch.randn(n, H * D, device=DEV).to(BF16)
    k, v = torch.ones(3, G, 384, D, device=DEV, dtype=BF16), torch.ones(3, G, 384, V, device=DEV, dtype=BF16)
    for slots, seen in ((3, 1.0), (2, 0.0)):
        out = torch.full((n, H * V), 7.0, device=DEV, dtype=BF16)
        nsq.attention(q, k[:slots], v[:slots], out, H, D ** -0.5, None, None, False, nsq.Batch([2], [0], [n], torch.device(DEV)), impl=impl)
        assert bool((out == seen).all())


@pytest.mark.gpu
@pytest.mark.parametrize("H,G,D,V,n,stored", [(2, 2, 96, 64, 150, 0), (2, 2, 96, 64, 80, 63), (4, 4, 72, 40, 300, 7), (4, 1, 136, 80, 700, 0)])
@pytest.mark.parametrize("window", [0, 1, 64])
def test_dense_rows_off_the_boxes(H, G, D, V, n, stored, window):
    """They take no tensor map: the form whose waits are made to run out (impl 3) has none."""
    from promptcache_b200 import _native_seq as nsq
    g = torch.Generator(device=DEV).manual_seed(D + n)
    cap = (n + stored + 63) // 64 * 64
    rnd = lambda *s: torch.randn(*s, generator=g, device=DEV).to(BF16)
    q, k, v, out = rnd(n, H * D), rnd(1, G, cap, D), rnd(1, G, cap, V), torch.full((n, H * V), 7.0, device=DEV, dtype=BF16)
    before = nsq.load().pcs_attn_timeouts()
    nsq.attention(q, k, v, out, H, D ** -0.5, None, None, False, nsq.Batch([1], [stored], [n], torch.device(DEV)), impl=3, window=window,
                  pool_slot=torch.zeros(1, dtype=torch.int32, device=DEV))
    assert nsq.load().pcs_attn_timeouts() == before
    i, j = torch.arange(stored, stored + n, device=DEV)[:, None], torch.arange(stored + n, device=DEV)[None]
    hidden = (j > i) | ((i - j >= window) if window else torch.zeros_like(j > i))
    for h in range(H):
        kk, vv = k[0, h * G // H, :n + stored].to(F64), v[0, h * G // H, :n + stored].to(F64)
        want = torch.softmax((q[:, h * D:(h + 1) * D].to(F64) @ kk.T * D ** -0.5).masked_fill(hidden, -torch.inf), -1) @ vv
        got = out[:, h * V:(h + 1) * V].to(F64)
        # the result is rounded to bfloat16 (2^-9 of it), the weights keep 16 bits and the scores 22
        assert bool(((got - want).abs() <= want.abs() * 2.0 ** -8 + vv.abs().max() * 2.0 ** -13).all()), h


@pytest.mark.gpu
@pytest.mark.parametrize("H,G,D,V,limits", [(2, 2, 96, 64, {}), (2, 1, 96, 64, dict(window=30)), (4, 2, 72, 136, dict(softcap=20.0)), (2, 2, 200, 40, dict(chunk=70))])
def test_hidden_rows_that_are_not_finite(H, G, D, V, limits):
    """A value of NaN or infinity reaches the queries that see its key and no others of their tile."""
    from promptcache_b200 import _native_seq as nsq
    n, stored, key = 150, 9, 100
    g = torch.Generator(device=DEV).manual_seed(D)
    rnd = lambda *s: torch.randn(*s, generator=g, device=DEV).to(BF16)
    q, k, v, batch = rnd(n, H * D), rnd(1, G, 192, D), rnd(1, G, 192, V), nsq.Batch([1], [stored], [n], torch.device(DEV))
    outs = []
    for value in (None, torch.nan, torch.inf):
        if value is not None:
            v[0, :, key] = value
        out = torch.full((n, H * V), 7.0, device=DEV, dtype=BF16)
        nsq.attention(q, k, v, out, H, D ** -0.5, None, None, False, batch, pool_slot=torch.zeros(1, dtype=torch.int32, device=DEV), **limits)
        outs.append(out)
    i = torch.arange(stored, stored + n, device=DEV)
    sees = (i >= key) & (i - key < limits.get("window", n)) & (i // limits.get("chunk", 10 ** 6) == key // limits.get("chunk", 10 ** 6))
    assert 0 < int(sees.sum()) < n
    for out in outs[1:]:
        # the same numbers summed in another order, rounded to bfloat16
        assert bool(((out[~sees].double() - outs[0][~sees].double()).abs() <= outs[0][~sees].double().abs() * 2.0 ** -7 + 2.0 ** -10).all())
        assert not bool(out[sees].isfinite().any())
