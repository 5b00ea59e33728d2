"""Which prompts of gated linear attention walk over their chunks in one launch: those that were measured to be faster so."""
import pytest

from promptcache_b200 import _native_seq as nsq


@pytest.mark.parametrize("lens,heads,dim,vdim,one", [   # us in one / as sums and a scan
    ((1500, 548), 4, 256, 512, True), ((4096,), 8, 256, 512, True), ((300, 300), 8, 256, 512, True), ((100,), 2, 64, 128, True),
    ((1024,), 8, 128, 256, False),     # 23.0 / 17.3
    ((1024,), 2, 256, 512, False),     # 23.0 / 17.6
    ((870,), 8, 128, 256, False),      # 20.4 / 16.6
    ((1063,), 2, 256, 512, False),     # 24.3 / 18.8
    ((2048,), 4, 128, 128, False), ((4096,), 2, 128, 256, False),
])
def test_states_in_one(lens, heads, dim, vdim, one):
    chunks = [-(-n // 64) for n in lens]
    assert nsq._gla_states_in_one(sum(chunks), max(chunks), heads, dim, vdim) is one
