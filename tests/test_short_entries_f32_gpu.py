"""Prompt attention in 32 bits over a few tokens and keys, with and without a workspace, where the launch chooses between kernels by size."""
import pytest

from tests.test_attention_bias_table_gpu import F32, nsq  # noqa: F401  (nsq: the fixture)
from tests.test_group_decode_gpu import check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name", ["plain", "window", "bias"])
@pytest.mark.parametrize("workspace", [False, True])
@pytest.mark.parametrize("lens,pos0", [((16,), (0,)), ((16,), (900,)), ((17, 40), (0, 20)), ((64,), (0,)), ((64,), (70,))])
def test_short_prompts_in_32_bits(nsq, lens, pos0, workspace, name):  # noqa: F811
    for H, G, D, V in ((4, 2, 128, 128), (2, 1, 36, 20)):
        check(nsq, name, H, G, D, V, lens, pos0, F32, workspace, D)
