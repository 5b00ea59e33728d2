"""Prompt attention over short entries, where the launch chooses between kernels by size: many entries of a few tokens, few of them, few and many keys."""
import pytest

from tests.test_attention_bias_table_gpu import BF16, nsq  # noqa: F401  (nsq: the fixture)
from tests.test_attention_forms_gpu import compare

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name", ["plain", "window", "chunk"])
@pytest.mark.parametrize("H,G,D,V,lens,pos0", [
    (16, 4, 64, 64, (64,) * 10 + (17, 1), (100,) * 12),     # many: 64 rows per block
    (4, 2, 64, 64, (33, 16), (0, 0)),                       # few over one key tile
    (4, 2, 64, 64, (33, 16), (700, 5)),                     # few over many: a walk shared by a cluster
    (40, 8, 128, 128, (20,) * 8, (0,) * 8),
    (8, 2, 128, 64, (128, 90), (0, 31)),
])
def test_short_prompts(nsq, H, G, D, V, lens, pos0, name):  # noqa: F811
    compare(nsq, name, BF16, H, G, D, V, lens, pos0)
