"""The chunked delta rule's launches refuse operands that their wide loads and stores could not reach, before anything is launched."""
import ctypes as C

import pytest

from promptcache_b200 import _native_seq as nsq

BASE = 1 << 20


def params(dtype, vdim, **fields):
    p, n = nsq.pcs_delta_chunk_params(), nsq.pcs_headnorm_params()
    for name, kind in p._fields_:
        if kind is C.c_void_p:
            setattr(p, name, BASE)
    for name in ("w", "g", "out"):
        setattr(n, name, BASE)
    p.heads = p.kv_heads = p.n_chunks = p.n_seqs = 1
    p.dim, p.vdim, p.n_tokens, p.dtype, p.parts = 64, vdim, 64, dtype, 2
    for name, value in fields.items():
        setattr(p, name, value)
    return p, n


@pytest.mark.parametrize("call,dtype,vdim,field,off", [
    ("prep", nsq.PCS_BF16, 64, "w", 8), ("prep", nsq.PCS_BF16, 64, "kd", 4), ("prep", nsq.PCS_BF16, 64, "u", 8), ("prep", nsq.PCS_BF16, 33, "w", 4), ("prep", nsq.PCS_F32, 64, "w", 4),
    ("scan", nsq.PCS_BF16, 64, "u", 4), ("scan", nsq.PCS_BF16, 6, "s", 4), ("scan", nsq.PCS_BF16, 64, "s_pool", 4), ("scan", nsq.PCS_BF16, 64, "kd", 8), ("scan", nsq.PCS_F32, 64, "w", 4),
    ("out", nsq.PCS_BF16, 64, "s", 8), ("out", nsq.PCS_BF16, 36, "u", 4), ("out", nsq.PCS_BF16, 33, "qd", 4),
])
def test_operands_off_their_pieces_are_refused(call, dtype, vdim, field, off):
    for per_head in (False, True):
        p, n = params(dtype, vdim, **{field: BASE + off}, **(dict(ld=None) if per_head else {}))
        args = (C.byref(p), C.byref(n), None) if call == "out" else (C.byref(p), None)
        assert getattr(nsq.load(), "pcs_delta_chunk_" + call)(*args) != 0
        text = nsq.load().pcs_last_error().decode()
        assert call in text and "-byte aligned" in text, text
