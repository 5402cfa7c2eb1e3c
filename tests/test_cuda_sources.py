"""Rules that the CUDA sources keep, checked as text and in what the compiler reports of the build."""
from __future__ import annotations

import glob
import os
import re

import pytest
from conftest import ROOT


def test_instructions_of_a_whole_warp_are_volatile():
    """An `asm` that is not volatile may move to where its result is used, into a branch that part of a warp takes.  Instructions that all lanes
    execute together (`.sync`) are undefined there, so each is volatile."""
    paths = sorted(glob.glob(os.path.join(ROOT, "trellis_serve_b200", "csrc", "*.cu*")))
    statements = [(os.path.basename(p), m) for p in paths for m in re.findall(r"(?s)\basm\b(\s*volatile)?\s*\((.*?)\)\s*;", open(p).read())]
    assert any(".sync" in text for _, (_, text) in statements)
    assert [(p, text[:40]) for p, (volatile, text) in statements if re.search(r"\.sync\b", text) and not volatile] == []


def test_decode_instances_of_one_or_two_rows_do_not_spill():
    """The launches of a decoded token are short: registers kept in memory by their epilogue showed as 12 % of the output projection."""
    log = os.path.join(ROOT, "trellis_serve_b200", "csrc", "build", "ptxas.log")
    if not os.path.exists(log):
        pytest.skip("no report of a build")
    found = re.findall(r"Compiling entry function '(\w*skinny_kernelILi\dELi\dELi\dELi2E\w*)'[^\n]*\n[^\n]*\n\s*(\d+) bytes stack frame, (\d+) bytes spill stores, (\d+) bytes",
                       open(log).read())
    assert len(found) >= 7 * 3 * 7                          # bit rates, codebook forms, sources of activations and epilogues
    assert [f for f in found if f[1:] != ("0", "0", "0")] == []
