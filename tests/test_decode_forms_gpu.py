"""Decoding attention at the sizes where its forms meet: clusters, splits through the workspace, a block per head."""
import pytest

from tests.test_attention_bias_table_gpu import BF16, F32, nsq  # noqa: F401  (nsq: the fixture)
from tests.test_group_decode_gpu import check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dt", [BF16, F32])
@pytest.mark.parametrize("H,G,D,V,pos0", [
    (4, 2, 128, 128, (3000,)),            # more splits than a cluster has
    (20, 1, 256, 256, (2000, 300)),       # three blocks per group, the last of four heads, in clusters
    (20, 1, 256, 256, (300,)),            # a block per head
    (16, 2, 64, 64, (130, 50)),
    (16, 2, 64, 64, (99, 127)),           # 128 keys at most
    (3, 1, 64, 64, (2500, 1)),
])
def test_decoding_forms(nsq, dt, H, G, D, V, pos0):  # noqa: F811
    if dt == F32 and D > 128:
        pytest.skip("wider than the kernel's rows in 32 bits")
    check(nsq, "bias", H, G, D, V, (1,) * len(pos0), pos0, dt, True, D)
