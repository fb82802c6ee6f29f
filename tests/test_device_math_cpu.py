"""Layouts and arithmetic of the kernels' headers, run on the host."""
import pytest

from device_math_build import load


@pytest.fixture(scope="module")
def dm(tmp_path_factory):
    return load(str(tmp_path_factory.mktemp("device_math")))


def test_an_fp32_outbox_entry_is_aligned_for_its_128_bit_accesses(dm):
    """k_insert copies an entry into a local one in two 128-bit halves"""
    assert dm.dm_out_mixed_size() == 32 and dm.dm_out_mixed_align() == 16
