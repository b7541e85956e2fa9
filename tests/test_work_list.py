"""The engine's kept work lists do not outlive the arena that holds them
(tests/work_list_check.cpp: an arena gets an earlier one's addresses)."""
import pytest

import host_check


@pytest.mark.skipif(not host_check.AVAILABLE, reason="needs g++, CUDA's headers")
def test_work_list_after_the_arena_grew(tmp_path):
    host_check.run(tmp_path, "work_list_check")
