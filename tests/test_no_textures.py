"""The boundary's calls are refused without the picture memory
(tests/no_textures_check.cpp)."""
import pytest

import host_check


@pytest.mark.skipif(not host_check.AVAILABLE, reason="needs g++, CUDA's headers")
def test_calls_without_textures_are_refused(tmp_path):
    host_check.run(tmp_path, "no_textures_check")
