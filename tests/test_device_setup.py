"""Kernel attributes belong to a device: what raises a kernel's shared memory in the slot-pool library is kept per device, never behind a flag of the process.  (Read from the sources: a
second device is not at hand where the tests run.)"""
import re
from pathlib import Path

import pytest

SOURCES = sorted((Path(__file__).parent.parent / "promptcache_b200" / "csrc").glob("seq_*.cu*"))


@pytest.mark.parametrize("path", SOURCES, ids=lambda p: p.name)
def test_no_flag_of_the_process(path):
    assert not re.findall(r"static (?:std::atomic<)?bool>? \w+(?: = |\{| ?;)", path.read_text())
