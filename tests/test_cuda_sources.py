"""Rules that the CUDA sources keep, checked as text."""
from __future__ import annotations

import glob
import os
import re

from conftest import ROOT


def test_instructions_of_a_whole_warp_are_volatile():
    """An `asm` that is not volatile may move to where its result is used, into a branch that part of a warp takes.  Instructions that all lanes
    execute together (`.sync`) are undefined there, so each is volatile."""
    paths = sorted(glob.glob(os.path.join(ROOT, "trellis_serve_b200", "csrc", "*.cu*")))
    statements = [(os.path.basename(p), m) for p in paths for m in re.findall(r"(?s)\basm\b(\s*volatile)?\s*\((.*?)\)\s*;", open(p).read())]
    assert any(".sync" in text for _, (_, text) in statements)
    assert [(p, text[:40]) for p, (volatile, text) in statements if re.search(r"\.sync\b", text) and not volatile] == []
