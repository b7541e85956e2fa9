"""Set-up written on the legacy stream is complete before the engine's and the
boundary's own streams use it (tests/setup_wait_check.cpp)."""
import pytest

import host_check


@pytest.mark.skipif(not host_check.AVAILABLE, reason="needs g++, CUDA's headers")
@pytest.mark.parametrize("part", ["engine", "boundary"])
def test_setup_is_complete_before_use(tmp_path, part):
    host_check.run(tmp_path, "setup_wait_check", part)
