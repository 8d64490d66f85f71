"""State that an entry point keeps between calls, read from the sources: callers come from several threads, and the binding
lets go of the GIL."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "nnabla_b200", "csrc")
SOURCES = sorted(glob.glob(os.path.join(CSRC, "*.cu")) + glob.glob(os.path.join(CSRC, "*.cuh")))


@pytest.mark.parametrize("path", SOURCES, ids=os.path.basename)
def test_variables_kept_between_calls_are_atomic_or_locked(path):
    """A static variable of a function is constant, atomic, its thread's own, or declared beside the mutex that is locked
    for it."""
    lines = re.sub(r"//[^\n]*", "", open(path).read()).split("\n")
    for i, line in enumerate(lines):
        kept = re.match(r"\s+static\s+(?!const\b|constexpr\b|thread_local\b|std::atomic<|std::mutex\b)[^()]*[;={]", line)
        if kept:
            assert re.match(r"\s+static std::mutex (\w+);", lines[i - 1]), line
            assert re.search(r"std::lock_guard<std::mutex> \w+\(", "\n".join(lines[i:i + 10])), line
