"""Sigmoids inside results that leave in bfloat16 are 32-bit ones: a result may be rounded the other way only where the exact one lies within their few roundings of a rounding boundary.
(With an exponential and a reciprocal that are 2^-18 off, dozens of the results here are beyond that.)"""
import ctypes as C

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV, BF16, F64 = torch.device("cuda:0"), torch.bfloat16, torch.float64


def beyond(got, want, rel):
    """Results further off than half of a bfloat16 step (2^-8 of the power of two below them) and rel of themselves."""
    want = want.abs()
    return int(((got.to(F64).abs() - want).abs() > 2.0 ** (want.log2().floor() - 8) + rel * want).sum())


def gates(*s):
    """bfloat16 numbers from -80 to -8: where a sigmoid takes the most bits of its argument, and no result is below the smallest normal number."""
    return (torch.rand(*s, generator=torch.Generator().manual_seed(s[0]), dtype=F64) * -72 - 8).to(BF16)


def weights(n):
    return (1 + torch.arange(n) / n).to(BF16)


@pytest.mark.parametrize("rows,ff", [(512, 128), (33, 2048)])
def test_silu(rows, ff):
    from promptcache_b200 import _native_seq as nsq
    z, u = gates(rows, ff), weights(128).repeat(ff // 128).expand(rows, ff)
    got = nsq.glu_mul(torch.cat([z, u], 1).to(DEV), ff).cpu()
    # the exponential, 1 + e, the divide and two products: 2^-23 and four times 2^-24
    assert beyond(got, z.to(F64) * torch.sigmoid(z.to(F64)) * u.to(F64), 2.0 ** -21) == 0


# Below, every column of a head is the same number before the norm, so that what the gate multiplies is known: 1 or -1, to the roundings of a sum of up to 512 equal squares (a thread
# adds eight, the rest in pairs: 2^-21 of it), of the mean, the root, the reciprocal and the product with it.
@pytest.mark.parametrize("n,V", [(400, 128), (512, 256), (700, 512)])
def test_matrix_memory(n, V):
    from promptcache_b200 import _native_seq as nsq
    g = torch.Generator().manual_seed(V)
    H, D = 1, 64
    rnd = lambda *s: torch.randn(*s, generator=g)
    z, w = gates(n, V), weights(128).repeat(V // 128)
    proj = torch.cat([rnd(n, 2 * D).to(BF16), rnd(n, 1).to(BF16).expand(n, V), z], 1).contiguous().to(DEV)
    s, nn, m = torch.zeros(1, H, D, V, device=DEV), torch.zeros(1, H, D, device=DEV), torch.zeros(1, H, device=DEV)
    out = torch.empty(n, V, device=DEV, dtype=BF16)
    nsq.mlstm_scan(proj, (0, D, 2 * D, 2 * D + V), rnd(n, H).to(DEV), torch.nn.functional.logsigmoid(rnd(n, H) + 3).to(DEV), w.to(DEV), out, s, nn, m, 0.0, nsq.Batch([0], [0], [n], DEV))
    assert beyond(out.cpu(), torch.sigmoid(z.to(F64)) * w.to(F64), 2.0 ** -20) == 0


@pytest.mark.parametrize("chunks,D,V", [(8, 64, 128), (40, 64, 256), (100, 32, 256), (160, 16, 512)])
@pytest.mark.parametrize("parts", [2, 3])
@pytest.mark.parametrize("silu", [0, 1])
def test_chunked_read_out(chunks, D, V, parts, silu):
    from promptcache_b200 import _native_seq as nsq
    g = torch.Generator(device=DEV).manual_seed(chunks + D)
    T = 64 * chunks
    rnd = lambda *s: torch.randn(*s, generator=g, device=DEV)
    qd, s, a, u = rnd(chunks, 64, D), rnd(chunks, D, 1).expand(chunks, D, V).contiguous(), rnd(chunks, 64, 64).tril(), rnd(chunks, 64, 1).to(BF16).float().expand(chunks, 64, V).contiguous()
    z, w, out = gates(T, V), weights(128).repeat(V // 128), torch.empty(T, V, device=DEV, dtype=BF16)
    z_d, w_d, first, lens = z.to(DEV), w.to(DEV), torch.arange(0, T, 64, dtype=torch.int32, device=DEV), torch.full((chunks,), 64, dtype=torch.int32, device=DEV)
    p, n = nsq.pcs_delta_chunk_params(), nsq.pcs_headnorm_params()
    p.heads, p.kv_heads, p.dim, p.vdim, p.n_chunks, p.n_tokens, p.dtype, p.n_seqs, p.parts = 1, 1, D, V, chunks, T, nsq.PCS_BF16, 1, parts
    p.chunk_first, p.chunk_len, p.qd, p.a, p.s, p.u = (t.data_ptr() for t in (first, lens, qd, a, s, u))
    n.w, n.g, n.g_stride, n.out, n.out_stride = w_d.data_ptr(), z_d.data_ptr(), V, out.data_ptr(), V
    n.n_tokens, n.heads, n.vdim, n.eps, n.out_scale, n.dtype, n.silu = T, 1, V, 0.0, 1.0, nsq.PCS_BF16, silu
    nsq._check(nsq.load().pcs_delta_chunk_out(C.byref(p), C.byref(n), nsq._stream()), "pcs_delta_chunk_out")
    want = torch.sigmoid(z.to(F64)) * w.to(F64)
    assert beyond(out.cpu(), want * z.to(F64) if silu else want, 2.0 ** -20) == 0
