"""The autotuner times every kernel shape once: of two equal shapes noise would pick
one, and with it the order in which a surrogate's anchors are sampled.
"""
import importlib

autotune = importlib.import_module("lklight-gpu_b200.autotune")


def test_candidates_are_different_kernel_shapes():
    # groups of 8 are searched two at a time (include/lkg.h, lkg_ctx_set_group)
    shapes = [(tile, 16 if group == 8 else group, cell, xsub) for tile, group, cell, xsub in autotune.CANDIDATES]
    assert len(set(shapes)) == len(shapes)
    assert all(tile in (64, 128, 256) and group in (4, 8, 16, 32) for tile, group, _, _ in autotune.CANDIDATES)
