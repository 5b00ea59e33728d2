"""The tcgen05 prompt attention kernel against float64: edges of its 128-query and 64-key tiles, the two ways of pairing tiles, walks split over a
cluster, every option it applies to a score, widths off the padded ones, and rows behind a sequence's end that hold NaN."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV, BF16, F64 = "cuda:0", torch.bfloat16, torch.float64


@pytest.fixture(scope="module")
def nsq():
    from promptcache_b200 import _native_seq
    _native_seq.load()
    return _native_seq


def reference(q, k, v, p0, scale, h, o):
    """One head of one entry in float64: q [n, D], k and v [p0 + n, *]."""
    i, j = torch.arange(p0, p0 + q.shape[0], device=DEV)[:, None], torch.arange(p0 + q.shape[0], device=DEV)[None]
    s = q @ k.T * scale
    if "head_scale" in o:
        s = s * o["head_scale"][h].to(F64)
    if "softcap" in o:
        s = o["softcap"] * torch.tanh(s / o["softcap"])
    if "r1" in o:
        s = s - o["r1"][h].to(F64) * torch.log1p(o["r2"][h].to(F64) * (i - j).clamp(min=0))
    if "bias_table" in o:
        s = s + o["bias_table"][h].to(F64)[(i - j).clamp(0, o["bias_table"].shape[1] - 1)]
    hidden = j > i
    if "window" in o:
        hidden = hidden | ((i - j >= o["window"]) & (j >= o.get("keep_first", 0)))
    if "chunk" in o:
        hidden = hidden | (i // o["chunk"] != j // o["chunk"])
    s = s.masked_fill(hidden, -math.inf)
    mx = s.max(-1, keepdim=True).values
    sink = o["sink_logit"][h].to(F64) if "sink_logit" in o else torch.zeros((), dtype=F64, device=DEV)
    if o.get("sink"):
        mx = torch.maximum(mx, sink)
    e = torch.exp(s - mx)
    return e @ v / (e.sum(-1, keepdim=True) + (torch.exp(sink - mx) if o.get("sink") else 0.0))


OPTIONS = {
    "plain": lambda H, T, g: {},
    "bias": lambda H, T, g: dict(r1=torch.rand(H, generator=g, device=DEV), r2=torch.rand(H, generator=g, device=DEV), sink=True),
    "window": lambda H, T, g: dict(softcap=20.0, window=100, keep_first=70),
    "window_only": lambda H, T, g: dict(window=65),
    "chunk": lambda H, T, g: dict(chunk=96, bias_table=torch.randn(H, 50, generator=g, device=DEV), head_scale=torch.rand(H, generator=g, device=DEV) + 0.5, out_scale=0.7),
    "gated": lambda H, T, g: dict(sink=True, sink_logit=torch.randn(H, generator=g, device=DEV), head_gate=torch.randn(T, H, generator=g, device=DEV).to(BF16)),
}
SHAPES = [  # heads, kv heads, dim, vdim, new tokens, stored tokens
    (4, 2, 128, 128, (128, 129, 16, 257), (0, 63, 64, 1)),       # neighbouring tiles
    (2, 1, 64, 64, (700,), (0,)),                                # tiles from both ends, an even number of them
    (3, 3, 192, 128, (200, 31), (1900, 2000)),                   # a walk shared by eight blocks, one of them with few tiles
    (2, 1, 72, 40, (40,), (700,)),                               # widths off the padded ones, clusters
    (8, 1, 128, 64, (1023, 1), (130, 5)),
]


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("name", OPTIONS)
def test_prompt_attention(nsq, shape, name):
    H, G, D, V, lens, pos0 = shape
    g = torch.Generator(device=DEV).manual_seed(len(name) * 100 + D)
    T, B, cap = sum(lens), len(lens), (max(n + p for n, p in zip(lens, pos0)) + 127) // 128 * 128
    q = (torch.randn(T, H * D, generator=g, device=DEV) * 2).to(BF16)
    k, v = torch.randn(B + 1, G, cap, D, generator=g, device=DEV).to(BF16), torch.randn(B + 1, G, cap, V, generator=g, device=DEV).to(BF16)
    slots = [B - b for b in range(B)]
    for b, (n, p) in enumerate(zip(lens, pos0)):
        k[slots[b], :, n + p:], v[slots[b], :, n + p:] = math.nan, math.nan
    o = OPTIONS[name](H, T, g)
    out = torch.full((T, H * V + 8), 7.0, device=DEV, dtype=BF16)
    opt = {a: x for a, x in o.items() if a not in ("r1", "r2", "sink")}
    for view in (out[:, :H * V], torch.empty(T, H * V, device=DEV, dtype=BF16)):   # a column range of a wider matrix, and a dense one
        nsq.attention(q, k, v, view, H, D ** -0.5, o.get("r1"), o.get("r2"), o.get("sink", False), nsq.Batch(slots, pos0, lens, torch.device(DEV)), **opt)
        off = 0
        for b, (n, p) in enumerate(zip(lens, pos0)):
            for h in range(H):
                kk, vv = k[slots[b], h * G // H, :n + p].to(F64), v[slots[b], h * G // H, :n + p].to(F64)
                want = reference(q[off:off + n, h * D:(h + 1) * D].to(F64), kk, vv, p, D ** -0.5, h, o) * o.get("out_scale", 1.0)
                if "head_gate" in o:
                    want = want * torch.sigmoid(o["head_gate"][off:off + n, h].to(F64))[:, None]
                got = view[off:off + n, h * V:(h + 1) * V].to(F64)
                # the result is rounded to bfloat16 (2^-9 of it), the weights keep 16 bits and the scores 22 (of up to 2^5 in the base-2 domain)
                bound = want.abs() * 2.0 ** -8 + vv.abs().max() * 2.0 ** -13
                assert bool(((got - want).abs() <= bound).all()), (b, h, float(((got - want).abs() - bound).max()))
            off += n
    assert bool((out[:, H * V:] == 7.0).all())
    assert nsq.load().pcs_attn_timeouts() == 0


def test_score_that_is_not_a_number_stays_visible(nsq):
    """A key row of NaN under a cap: every query that sees it gets NaN, queries of earlier tiles do not."""
    g = torch.Generator(device=DEV).manual_seed(1)
    q, k, v = (torch.randn(*s, generator=g, device=DEV).to(BF16) for s in ((300, 128), (1, 1, 384, 128), (1, 1, 384, 128)))
    k[0, 0, 200] = math.nan
    out = torch.empty(300, 128, device=DEV, dtype=BF16)
    nsq.attention(q, k, v, out, 1, 128 ** -0.5, None, None, False, nsq.Batch([0], [0], [300], torch.device(DEV)), softcap=30.0)
    assert bool(out[200:].isnan().all()) and not bool(out[:192].isnan().any())
