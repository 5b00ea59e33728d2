"""A chunk's preparation for the delta rule (bfloat16 runs, decays per channel or per head) against float64: the sums over pairs, the solved values and keys, the outgoing keys, at the edges of its tiles
(four channels, eight, sixteen tokens, 32 columns), with strong decays, none at all, and values whose rows start off eight bytes."""
import ctypes as C

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV, BF16, F32, F64 = torch.device("cuda:0"), torch.bfloat16, torch.float32, torch.float64


@pytest.mark.parametrize("KV,G,D,V,lens,rate", [
    (1, 1, 4, 4, (1, 64), 1.0), (1, 2, 20, 33, (15, 17), 0.1), (2, 1, 36, 40, (64, 33), 20.0), (1, 1, 100, 7, (63, 16, 49), 0.0), (2, 2, 128, 128, (64, 31), 1.0), (1, 2, 256, 512, (64, 50), 0.5),
    (1, 1, 7, 65, (40,), 1.0),
])
@pytest.mark.parametrize("per_head", [False, True])
def test_prep(KV, G, D, V, lens, rate, per_head):
    from promptcache_b200 import _native_seq as nsq
    g = torch.Generator().manual_seed(D * 3 + V)
    H, T, nc = KV * G, sum(lens), len(lens)
    first = [sum(lens[:i]) for i in range(nc)]
    unit = lambda x: x / x.norm(dim=-1, keepdim=True)
    q, k = unit(torch.randn(T, KV, D, generator=g)), unit(torch.randn(T, KV, D, generator=g))
    qk = torch.cat([q.reshape(T, -1), k.reshape(T, -1)], 1).contiguous()
    v = torch.randn(T, H * V, generator=g).to(BF16)
    ld = -rate * torch.rand(T, H, D, generator=g) * torch.rand(T, H, D, generator=g)
    b = torch.randn(T, H, generator=g).to(BF16)
    dec_a, bias, rates = torch.randn(T, H, generator=g).to(BF16), torch.randn(H, generator=g) * 0.5, rate * (0.2 + torch.rand(H, generator=g))
    if per_head:
        ld = (-rates.to(F64) * torch.nn.functional.softplus(dec_a.to(F64) + bias.to(F64)))[:, :, None].expand(T, H, D)
        rate = float(ld.abs().max())
    D8, L = (D + 7) // 8 * 8, (D + 63) // 64 * 64
    dev = {n: t.to(DEV).contiguous() for n, t in dict(qk=qk, v=v, ld=ld.float(), b=b, dec_a=dec_a, bias=bias, rates=rates, first=torch.tensor(first, dtype=torch.int32), lens=torch.tensor(lens, dtype=torch.int32)).items()}
    o = {n: torch.full(s, 7.0, device=DEV) for n, s in dict(qd=(nc * H, 64, D), kd=(nc * H, 64 * L), w=(nc * H, D8 * 64), g=(nc * H, D), u=(nc * H, 64, V), a=(nc * H, 64, 64)).items()}
    p = nsq.pcs_delta_chunk_params()
    p.qk, p.v, p.ld, p.b, p.b_stride = (dev["qk"].data_ptr(), dev["v"].data_ptr(), dev["ld"].data_ptr(), dev["b"].data_ptr(), H)
    if per_head:
        p.ld, p.dec_a, p.dec_stride, p.dt_bias, p.rate = None, dev["dec_a"].data_ptr(), H, dev["bias"].data_ptr(), dev["rates"].data_ptr()
    p.heads, p.kv_heads, p.dim, p.vdim, p.n_chunks, p.n_tokens, p.dtype, p.n_seqs = H, KV, D, V, nc, T, nsq.PCS_BF16, 1
    p.chunk_first, p.chunk_len = dev["first"].data_ptr(), dev["lens"].data_ptr()
    p.qd, p.kd, p.w, p.g, p.u, p.a = (o[n].data_ptr() for n in ("qd", "kd", "w", "g", "u", "a"))
    nsq._check(nsq.load().pcs_delta_chunk_prep(C.byref(p), nsq._stream()), "pcs_delta_chunk_prep")
    got = {n: t.cpu().to(F64) for n, t in o.items()}
    # place x of w's tile of eight is channel (x >> 1) + 4 (x & 1); a lane holds rows g, g + 8 of places 2 t, 2 t + 1
    w = torch.zeros(nc * H, 64, D8, dtype=F64)
    f = got["w"].view(nc * H, D8 // 8, 4, 8, 4, 2, 2)     # tile, rows' tile, g, t, place's low bit, row's upper half
    for x in range(2):
        for t in range(4):
            c = t + 4 * x
            w[:, :, c::8] = f[:, :, :, :, t, x, :].permute(0, 2, 4, 3, 1).reshape(nc * H, 64, D8 // 8)
    # kd's tile of 16 channels and 8 tokens: a lane holds channels g, g + 8 of tokens t, t + 4
    kd = got["kd"].view(nc * H, L // 16, 8, 8, 4, 2, 2).permute(0, 2, 5, 4, 1, 6, 3).reshape(nc * H, 64, L)
    # 2^-22 of an exponential, 2^-24 of each of the up to 64 numbers a running sum holds (64 rate each) and of the up to 256 terms of a sum; the solve adds 64 terms three times over
    eps = 2.0 ** -22 * (1 + 64 * rate) + 2.0 ** -23 * (16 + D ** 0.5)
    for c in range(nc):
        n, sl = lens[c], slice(first[c], first[c] + lens[c])
        for h in range(H):
            B = ld[sl, h].to(F64).cumsum(0)
            E = torch.exp((B[:, None] - B[None]).clamp(max=0))
            qf, kf = q[sl, h // G].to(F64), k[sl, h // G].to(F64)
            aq = torch.einsum("id,sd,isd->is", qf, kf, E).tril()
            ak = torch.einsum("id,sd,isd->is", kf, kf, E).tril(-1)
            beta = torch.sigmoid(b[sl, h].to(F64))
            inv = torch.linalg.inv(torch.eye(n, dtype=F64) + beta[:, None] * ak)
            size = float(inv.abs().sum(1).max()) ** 2
            u, wk = inv @ (beta[:, None] * v[sl, h * V:(h + 1) * V].to(F64)), inv @ (beta[:, None] * kf * torch.exp(B))
            j = c * H + h
            assert float((got["a"][j, :n, :n] - aq).abs().max()) <= 4 * eps
            assert bool((got["a"][j].triu(1) == 0).all())
            assert float((got["u"][j, :n] - u).abs().max()) <= 4 * eps * size * float(v.float().abs().max())
            assert float((w[j, :n, :D] - wk).abs().max()) <= 4 * eps * size
            assert float((got["qd"][j, :n] - qf * torch.exp(B)).abs().max()) <= eps
            assert float((got["g"][j] - torch.exp(B[-1])).abs().max()) <= eps
            assert float((kd[j, :n, :D] - kf * torch.exp(B[-1] - B)).abs().max()) <= eps
            assert bool((kd[j, n:] == 0).all()) and bool((kd[j, :, D:] == 0).all())
