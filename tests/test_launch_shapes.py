"""The launchers refuse what no kernel is built for, before they launch anything:
a group size without an instantiation (its spheres and strides would be read as
another size's) and per-atom outputs in the f64 mode (they would stay unwritten).
"""
import ctypes
import os
import subprocess

import pytest

from tests.lkg_helpers import REPO, lkg

INVALID_VALUE = 1   # cudaErrorInvalidValue

SHIM = r"""
#include "lkg_internal.h"
extern "C" int shape(int kind, int group, int tile, int atoms) {
    lkg::LaunchParams p{};
    float dummy = 0.f;
    p.group = group;
    p.tile = tile;
    p.atom_elec = atoms ? &dummy : nullptr;
    switch (kind) {
        case 0: return (int)lkg::launch_score_fast(p, 128, 1, nullptr);
        case 1: return (int)lkg::launch_score_exact(p, 1, nullptr);
        default: return (int)lkg::launch_desolv_fast(p, 512, 1, 64, nullptr);
    }
}
"""


@pytest.fixture(scope="module")
def shape(tmp_path_factory):
    lkg.lib()
    d = tmp_path_factory.mktemp("shape")
    src, so = str(d / "shape.cpp"), str(d / "shape.so")
    with open(src, "w") as f:
        f.write(SHIM)
    lib = os.path.join(REPO, "lklight-gpu_b200", "lib")
    subprocess.run(["g++", "-std=c++17", "-shared", "-fPIC", "-I" + os.path.join(REPO, "lklight-gpu_b200", "csrc"),
                    "-I/usr/local/cuda/include", src, "-o", so, "-L" + lib, "-Wl,-rpath," + lib, "-l:liblkg.so"],
                   check=True)
    return ctypes.CDLL(so).shape


# (eights have a cpydock kernel only)
@pytest.mark.parametrize("kind,group", [(k, g) for k in (0, 1, 2) for g in (0, 2, 8, 24, 64) if (k, g) != (2, 8)])
def test_group_sizes_without_a_kernel(shape, kind, group):
    assert shape(kind, group, 192, 0) == INVALID_VALUE


@pytest.mark.parametrize("kind,group,tile", [(0, 16, 40), (1, 16, 40), (0, 32, 48), (1, 32, 48)])
def test_tiles_of_broken_groups(shape, kind, group, tile):
    assert shape(kind, group, tile, 0) == INVALID_VALUE


def test_per_atom_outputs_in_the_f64_mode(shape):
    assert shape(1, 16, 128, 1) == INVALID_VALUE
