"""The per-family kernel libraries hold every function that their sources call."""
import os
import re

import pytest

from tensorrt_edge_llm_b200 import build


def _source(name):
    with open(os.path.join(build.CSRC, "kernels", name)) as f:
        return re.sub(r'//[^\n]*|"(?!C")[^"\n]*"', "", f.read())


@pytest.mark.parametrize("family", sorted(build.KERNEL_SETS))
def test_family_sources_are_closed_under_calls(family):
    """Unresolved symbols keep the library from loading, and with it the family on a machine without the whole library."""
    text = [_source(f) for f in build.KERNEL_SETS[family]]
    defined = {n for t in text for n in re.findall(r'extern "C"[^;{]*?\b(telb_\w+)\s*\([^;{]*\)\s*\{', t)}
    called = {n for t in text for n in re.findall(r"\b(telb_\w+)\s*\(", t)}
    assert defined and not called - defined
