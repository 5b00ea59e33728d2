"""One token of more than sixteen sequences, with a workspace and without one, and a workspace that is smaller than the decoding kernels ask for."""
import pytest

from tests.test_attention_bias_table_gpu import BF16, F32, nsq  # noqa: F401  (nsq: the fixture)
from tests.test_group_decode_gpu import check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dt", [BF16, F32])
@pytest.mark.parametrize("workspace", [True, False])
@pytest.mark.parametrize("n,H,G,D,V", [(17, 4, 1, 128, 128), (40, 2, 2, 64, 36), (70, 9, 1, 72, 64)])
def test_more_than_sixteen_sequences(nsq, dt, workspace, n, H, G, D, V):  # noqa: F811
    check(nsq, "bias", H, G, D, V, (1,) * n, tuple(range(0, 37 * n, 37)), dt, workspace, n)


def test_prompt_of_sixteen_tokens_with_a_small_workspace(nsq):  # noqa: F811
    check(nsq, "plain", 4, 2, 128, 128, (16,), (900,), F32, 8, 1)
