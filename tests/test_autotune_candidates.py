"""The autotuner times every kernel shape once: of two equal shapes noise would pick
one, and with it the order in which a surrogate's anchors are sampled.
"""
import importlib

import numpy as np
import pytest

autotune = importlib.import_module("lklight-gpu_b200.autotune")


@pytest.mark.parametrize("family,n_lig", [("dna", 300), ("vdw", 5000), ("cpydock", 300), ("cpydock", 5000)])
def test_candidates_are_different_kernel_shapes(family, n_lig):
    # groups of 8 are searched two at a time, but for small cpydock ligands
    # (include/lkg.h, lkg_ctx_set_group)
    items = [dict(family=family, lig=dict(coords=np.zeros((n_lig, 3))))]
    eights = family == "cpydock" and n_lig <= 700
    cand = autotune.candidates_for(items)
    shapes = [(tile, 16 if group == 8 and not eights else group, cell, xsub) for tile, group, cell, xsub in cand]
    assert len(set(shapes)) == len(shapes)
    assert all(tile in (64, 128, 256) and group in (4, 8, 16, 32) for tile, group, _, _ in cand)
    assert any(group == 8 for _, group, _, _ in cand) == eights
