"""The panel's exchange slots: data and tag of a word have to arrive together.
PTX makes no promise across the elements of a vector access, only within one,
so every vector access to a slot is made of 64-bit elements."""
import os
import re

import lila_gb300


def test_tagged_words_are_single_accesses():
    src = open(os.path.join(os.path.dirname(lila_gb300.__file__), "csrc", "lg_panel.cu")).read()
    kinds = re.findall(r"\b(?:ld|st)\.volatile\.global\.(\S+)", src)
    assert len(kinds) >= 2
    assert all(re.fullmatch(r"(v2\.)?[bus]64", k) for k in kinds), kinds
