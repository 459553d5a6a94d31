"""bench.py divides counted visits by timed passes: both have to be of the same
traversal variant."""
import os
import sys

import pytest

ROOT = os.path.abspath(os.path.join(os.path.dirname(__file__), ".."))
sys.path.insert(0, ROOT)
import bench  # noqa: E402


@pytest.mark.parametrize("traversal,ties,kernel,counted", [
    (0, 0, "k_wf_extend", 0), (0, 13, "k_wf_extend_pww", 3), (1, 0, "k_wf_extend_dyn", 1),
    (2, 13, "k_wf_extend_pww", 2), (3, 13, "k_wf_extend_pww", 3), (4, 0, "k_wf_extend", 4)])
def test_counts_are_of_the_timed_variant(traversal, ties, kernel, counted):
    tuning = {"block_trace": 64, "traversal": traversal, "refill_closest": 28}
    name, t = bench.timed_variant(tuning, {"ties": (0.1 * ties, ties)})
    assert name == kernel
    assert t == dict(tuning, traversal=counted) and tuning["traversal"] == traversal
