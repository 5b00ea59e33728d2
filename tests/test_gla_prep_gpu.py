"""A chunk's preparation in blocks of sixteen tokens against the general one (which the same call takes when a row starts off its pieces), and a read-out that takes the values
from the projections against one on their copies: sizes off the tiles, short chunks, decays that close within a token and ones that never do."""
import ctypes as C

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV, BF16, F32 = torch.device("cuda:0"), torch.bfloat16, torch.float32


def _prep(nsq, plan, batch, proj, shift, offs, ld, H, D, V, values=True):
    nc, T = plan["n_chunks"], proj.shape[0]
    wide = torch.zeros(T, proj.shape[1] + 8, device=DEV, dtype=BF16)
    wide[:, shift:shift + proj.shape[1]] = proj
    o = {k: torch.full(s, 7.0, device=DEV) for k, s in dict(qd=(nc * H, 64, D), kd=(nc * H, 64, D), g=(nc * H, D), vf=(nc * H, 64, V), a=(nc * H, 64, 64)).items()}
    p = nsq.pcs_gla_chunk_params()
    p.proj, p.row_stride = wide.data_ptr(), wide.stride(0)
    p.q_off, p.k_off, p.v_off, p.g_off = (x + shift for x in offs)
    p.ld, p.heads, p.dim, p.vdim, p.chunk, p.q_scale = ld.data_ptr(), H, D, V, 64, D ** -0.5
    p.chunk_first, p.chunk_len, p.n_chunks, p.n_tokens, p.dtype, p.n_seqs = plan["first"].data_ptr(), plan["len"].data_ptr(), nc, T, nsq.PCS_BF16, batch.n_seqs
    p.qd, p.kd, p.g, p.a = (o[k].data_ptr() for k in ("qd", "kd", "g", "a"))
    p.vf = o["vf"].data_ptr() if values else None
    nsq._check(nsq.load().pcs_gla_chunk_prep(C.byref(p), nsq._stream()), "pcs_gla_chunk_prep")
    return o, wide


@pytest.mark.parametrize("H,D,V,lens,rate", [
    (2, 4, 8, (1, 64), 1.0), (1, 20, 36, (15, 16, 17), 0.1), (2, 48, 64, (65, 33), 30.0), (3, 132, 72, (130, 7), 0.0), (1, 256, 512, (200, 49), 1.0), (2, 128, 128, (63, 48), 5.0),
    (1, 20, 36, (64, 61), 0.05), (2, 132, 72, (64,), 0.02), (1, 256, 512, (128, 50), 0.1),     # factors between blocks well away from 0 and 1
])
def test_blocks_of_sixteen(H, D, V, lens, rate):
    from promptcache_b200 import _native_seq as nsq
    g = torch.Generator().manual_seed(D + V)
    T = sum(lens)
    batch = nsq.Batch(list(range(len(lens))), [0] * len(lens), list(lens), DEV)
    plan = nsq._gla_chunk_plan(batch, 64)
    offs = (0, H * D, 2 * H * D, 2 * H * D + H * V)
    proj = torch.randn(T, 2 * H * D + 2 * H * V, generator=g).to(BF16).to(DEV)
    ld = (-rate * torch.rand(T, H, D, generator=g) * torch.rand(T, H, D, generator=g)).to(DEV)
    new, _ = _prep(nsq, plan, batch, proj, 0, offs, ld, H, D, V)
    old, _ = _prep(nsq, plan, batch, proj, 1, offs, ld, H, D, V)
    lean, _ = _prep(nsq, plan, batch, proj, 0, offs, ld, H, D, V, values=False)
    assert torch.equal(new["vf"], old["vf"]) and bool((lean["vf"] == 7.0).all())
    # a factor's logarithm is a difference of running sums of up to 64 numbers <= rate: both ways lose up to 64 of their roundings, 2^-24 of 64 * rate; sums of up to D products
    # lose less than D of theirs (bounded by the sums of absolute values)
    rel = 2.0 ** -24 * (64 * 64 * rate + 64)
    for k in ("qd", "kd", "g"):
        assert torch.equal(new[k], lean[k])
        assert float((new[k] - old[k]).abs().max()) <= rel * float(old[k].abs().max()), k
    assert torch.equal(new["a"], lean["a"])
    size = float(proj[:, :H * D].float().abs().max() * proj[:, H * D:2 * H * D].float().abs().max()) * D ** 0.5
    assert float((new["a"] - old["a"]).abs().max()) <= (rel + D * 2.0 ** -24) * size
    assert bool((new["a"].triu(1) == 0).all())
    # Every pair against float64: a factor is a product of up to four exponentials (2^-22 and a rounding each) of sums of up to sixteen numbers <= rate (sixteen roundings of numbers of up to
    # 16 rate, three such sums at most), a sum of D products loses less than D roundings of what its terms add up to in size
    rel = 2.0 ** -19 + 2.0 ** -24 * (3 * 16 * 16 * rate + D)
    first, lens_of = plan["first"].tolist(), plan["len"].tolist()
    for c in range(plan["n_chunks"]):
        sl = slice(first[c], first[c] + lens_of[c])
        for h in range(H):
            B = ld[sl, h].double().cumsum(0)
            q, k = (proj[sl, o + h * D:o + (h + 1) * D].double() for o in offs[:2])
            E = torch.exp((B[:, None] - B[None]).clamp(max=0))
            want, size = (torch.einsum("id,sd,isd->is", x * D ** -0.5, y, E).tril() for x, y in ((q, k), (q.abs(), k.abs())))
            assert bool(((new["a"][c * H + h, :lens_of[c], :lens_of[c]].double() - want).abs() <= rel * size + 1e-30).all()), (c, h)


@pytest.mark.parametrize("H,D,V,lens", [(2, 16, 8, (65, 1)), (1, 48, 136, (64, 33, 31)), (2, 256, 512, (130,)), (3, 64, 40, (17, 95))])
def test_values_in_place(H, D, V, lens):
    from promptcache_b200 import _native_seq as nsq
    g = torch.Generator().manual_seed(D + V)
    T = sum(lens)
    batch = nsq.Batch(list(range(len(lens))), [0] * len(lens), list(lens), DEV)
    plan = nsq._gla_chunk_plan(batch, 64)
    offs, nc = (0, H * D, 2 * H * D, 2 * H * D + H * V), plan["n_chunks"]
    proj = torch.randn(T, 2 * H * D + 2 * H * V, generator=g).to(BF16).to(DEV)
    ld = (-torch.rand(T, H, D, generator=g)).to(DEV)
    o, wide = _prep(nsq, plan, batch, proj, 0, offs, ld, H, D, V)
    s, w = torch.randn(nc * H, D, V, generator=g).to(DEV), torch.ones(V, device=DEV, dtype=BF16)
    outs = []
    for copies in (True, False):
        out = torch.zeros(T, H * V, device=DEV, dtype=BF16)
        r, n = nsq.pcs_delta_chunk_params(), nsq.pcs_headnorm_params()
        r.heads, r.kv_heads, r.dim, r.vdim, r.n_chunks, r.n_tokens, r.dtype, r.n_seqs, r.parts = H, H, D, V, nc, T, nsq.PCS_BF16, len(lens), 3
        r.chunk_first, r.chunk_len, r.qd, r.a, r.s = plan["first"].data_ptr(), plan["len"].data_ptr(), o["qd"].data_ptr(), o["a"].data_ptr(), s.data_ptr()
        r.u = o["vf"].data_ptr() if copies else None
        r.v, r.v_stride = wide.data_ptr() + 2 * offs[2], wide.stride(0)
        n.w, n.g, n.g_stride, n.out, n.out_stride = w.data_ptr(), wide.data_ptr() + 2 * offs[3], wide.stride(0), out.data_ptr(), out.stride(0)
        n.n_tokens, n.heads, n.vdim, n.eps, n.out_scale, n.dtype, n.silu = T, H, V, 1e-5, 1.0, nsq.PCS_BF16, 1
        nsq._check(nsq.load().pcs_delta_chunk_out(C.byref(r), C.byref(n), nsq._stream()), "pcs_delta_chunk_out")
        outs.append(out)
    assert torch.equal(*outs)     # the copies' lower parts are zeros
