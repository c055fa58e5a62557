"""bench.py's recorded instruction counts hold for the sources whose digest stands beside them: the
digest covers every file that the path kernel is compiled from, and the rule that cuts contracts
into its items.
"""
from __future__ import annotations

import os
import re

import bench

CSRC = os.path.join(bench.ROOT, "derivative-pricing_gb300", "csrc")


def _included(name, seen):
    seen.add(name)
    with open(os.path.join(CSRC, name)) as f:
        for inner in re.findall(r'^#include "([^"]+)"', f.read(), flags=re.M):
            if inner not in seen and os.path.exists(os.path.join(CSRC, inner)):
                _included(inner, seen)
    return seen


def test_digest_covers_what_the_path_kernel_is_made_of():
    want = _included("gbm_paths.cu", {"items.hpp"})
    assert {os.path.basename(p) for p in bench.PATH_KERNEL_SOURCES} >= want
    assert len(want) >= 6  # the includes were found


def test_recorded_counts_are_of_these_sources():
    assert bench.sources_digest() == bench.PATH_KERNEL_PROFILE["sources"]
