"""The slot-pool library's ctypes bindings: every entry with arguments declares them (an undeclared stream handle would pass as 32 bits)."""
import pytest

from promptcache_b200 import _native_seq as nsq

NO_ARGUMENTS = {"pcs_version", "pcs_last_error", "pcs_launch_count", "pcs_attn_timeouts"}


@pytest.mark.parametrize("name", nsq.EXPORTS)
def test_entry_declares_its_arguments(name):
    fn = getattr(nsq.load(), name)
    assert name in NO_ARGUMENTS or fn.argtypes, name


def test_scratch_size_is_64_bits():
    # one head of 256 x 512 states per chunk: 64 Mi tokens are far more than 2^31 floats
    assert nsq.load().pcs_mlstm_scratch_floats(1 << 26, 1, 8, 256, 512) > 1 << 32
