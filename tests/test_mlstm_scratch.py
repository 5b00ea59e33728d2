"""What the matrix-memory recurrence asks its caller for: scratch where its chunks run side by side, none where they never do."""
import pytest

from promptcache_b200 import _native_seq as nsq


def wanted(max_len, vdim, dim=64, dtype=nsq.PCS_BF16, impl=0, heads=2, n_seqs=3):
    p = nsq.pcs_mlstm_params()
    p.proj = p.norm_w = p.out = p.s_pool = 1 << 20
    p.heads, p.dim, p.vdim, p.n_seqs, p.n_tokens, p.max_len, p.dtype, p.impl = heads, dim, vdim, n_seqs, max_len, max_len, dtype, impl
    p.row_stride, p.q_off, p.k_off, p.v_off, p.g_off = 4096, 0, 512, 1024, 2048
    floats = nsq.load().pcs_mlstm_scratch_wanted(p)
    assert floats in (0, nsq.load().pcs_mlstm_scratch_floats(max_len, n_seqs, heads, dim, vdim))
    return floats > 0


@pytest.mark.parametrize("max_len,vdim,yes", [(192, 256, False), (193, 256, True), (448, 264, False), (449, 264, True), (448, 512, False), (449, 512, True), (5000, 520, False)])
def test_scratch_is_asked_for_where_it_is_used(max_len, vdim, yes):
    assert wanted(max_len, vdim) is yes


def test_other_forms_ask_for_none():
    assert not wanted(1000, 128, dtype=nsq.PCS_F32) and not wanted(1000, 128, impl=1) and not wanted(1000, 128, impl=2)
    assert not wanted(1000, 128, dim=72) and not wanted(1000, 128, dim=272) and not wanted(1000, 128, heads=65535, n_seqs=2)


@pytest.mark.parametrize("max_len,heads,n_seqs,dim,vdim,cut", [(384, 4, 4, 128, 256, False), (2048, 4, 1, 256, 512, False), (5000, 8, 3, 128, 256, False), (512, 2, 1, 64, 128, False),
                                                               (640, 2, 1, 64, 128, True), (1536, 37, 1, 64, 128, True), (1536, 38, 1, 64, 128, False)])
def test_room_for_segments_where_a_walk_has_some(max_len, heads, n_seqs, dim, vdim, cut):
    """What segments add up to takes 2.5 MB: asked for where the walk is cut, and not elsewhere."""
    p = nsq.pcs_mlstm_params()
    p.proj = p.norm_w = p.out = p.s_pool = 1 << 20
    p.heads, p.dim, p.vdim, p.n_seqs, p.n_tokens, p.max_len, p.dtype = heads, dim, vdim, n_seqs, 2 * max_len, max_len, nsq.PCS_BF16
    p.row_stride, p.q_off, p.k_off, p.v_off, p.g_off = 4096, 0, 512, 1024, 2048
    states = (2 * max_len // 64 + n_seqs) * heads * (dim * vdim + dim + 5 * 64 + 1) + n_seqs
    floats, most = nsq.load().pcs_mlstm_scratch_wanted(p), nsq.load().pcs_mlstm_scratch_floats(2 * max_len, n_seqs, heads, dim, vdim)
    assert floats == (states + 3) // 4 * 4 + (148 * 64 * 65 if cut else 0) and most >= floats
