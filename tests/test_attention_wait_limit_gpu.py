"""The tcgen05 prompt attention kernel when its waits run out: the launch ends, blocks are counted, and results are right all the same.  In a process of its own,
because the count belongs to the process."""
import multiprocessing
import traceback

import pytest
import torch

from tests.test_attention_bias_table_gpu import BF16, DEV, F64, bound, reference

pytestmark = pytest.mark.gpu
SHAPES = [  # heads, kv heads, dim, vdim, new tokens, stored tokens
    (4, 2, 128, 128, (128, 129, 16, 257), (0, 63, 64, 1)),       # neighbouring tiles
    (16, 4, 128, 128, (1500,), (0,)),                            # tiles from both ends
    (3, 3, 192, 128, (200, 31), (1900, 2000)),                   # a walk shared by eight blocks
    (2, 1, 72, 40, (40,), (700,)),
]
OPTIONS = ({}, dict(softcap=20.0, window=100, keep_first=70))


def _run(queue):
    from promptcache_b200 import _native_seq as nsq
    try:
        counts = []
        for H, G, D, V, lens, pos0 in SHAPES:
            for o in OPTIONS:
                g = torch.Generator(device=DEV).manual_seed(D + H)
                T, B, cap = sum(lens), len(lens), (max(n + p for n, p in zip(lens, pos0)) + 127) // 128 * 128
                q = (torch.randn(T, H * D, generator=g, device=DEV) * 2).to(BF16)
                k, v = torch.randn(B, G, cap, D, generator=g, device=DEV).to(BF16), torch.randn(B, G, cap, V, generator=g, device=DEV).to(BF16)
                out, batch = torch.full((T, H * V), 7.0, device=DEV, dtype=BF16), nsq.Batch(range(B), pos0, lens, torch.device(DEV))
                for impl in (3, 0):
                    nsq.attention(q, k, v, out, H, D ** -0.5, None, None, False, batch, impl=impl, **o)
                    counts.append(nsq.load().pcs_attn_timeouts())
                    off = 0
                    for b, (n, p) in enumerate(zip(lens, pos0)):
                        for h in range(H):
                            kk, vv = k[b, h * G // H, :n + p].to(F64), v[b, h * G // H, :n + p].to(F64)
                            want = reference(q[off:off + n, h * D:(h + 1) * D].to(F64), kk, vv, p, D ** -0.5, h, o)
                            got = out[off:off + n, h * V:(h + 1) * V].to(F64)
                            assert bool(((got - want).abs() <= bound(want, vv, BF16)).all()), (H, D, o, impl, b, h)
                        off += n
        queue.put(counts)
    except BaseException:
        queue.put(traceback.format_exc())


def test_waits_that_run_out():
    ctx = multiprocessing.get_context("spawn")
    queue = ctx.Queue()
    child = ctx.Process(target=_run, args=(queue,))
    child.start()
    counts = queue.get(timeout=240)
    child.join(60)
    assert isinstance(counts, list), counts
    hurried, patient = counts[::2], counts[1::2]
    assert hurried == patient and hurried[0] > 0      # waits of the usual length never run out
    assert all(a < b for a, b in zip(hurried, hurried[1:]))
