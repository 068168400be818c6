"""The warp kernels' candidate lists (one per 4 ligand atoms) at the sizes
where they can go wrong: ligands of one atom to a few groups with a ragged
last quad, every group size, and a receptor so dense that every list is
scored and refilled several times; against the oracle.

Tolerance: a pair's electrostatic term is clamped to 1 kcal/mol and its LJ term
to 1, so a pose of np near pairs adds at most 2 np + its clash sum (bounded by
|vdW part| + np) in absolute value; each term is computed in about a dozen f32
operations, 1e-6 relative.  Near-pair counts are exact.
"""
import numpy as np
import pytest

import oracle
from tests.lkg_helpers import lkg, random_poses

pytestmark = pytest.mark.gpu


def _molecule(coords, seed):
    rng = np.random.default_rng(seed)
    n = len(coords)
    return dict(coords=np.asarray(coords, np.float32).astype(np.float64), ele=rng.uniform(-0.8, 0.8, n),
                vdw=rng.uniform(0.015, 0.25, n), radius=rng.uniform(0.6, 2.1, n),
                heavy=rng.integers(0, 2, n).astype(np.uint8), hyd=rng.integers(0, 2, n).astype(np.int32),
                des=rng.uniform(-0.1, 0.1, n), asa=rng.uniform(-1.0, 70.0, n))


def _dense_receptor():
    g = np.arange(-8, 9) * 2.15   # 17^3 atoms, 0.1 per cubic A
    p = np.stack(np.meshgrid(g, g, g, indexing="ij"), -1).reshape(-1, 3)
    return _molecule(p + np.random.default_rng(1).uniform(-0.3, 0.3, p.shape), 2)


def _ligand(n):
    rng = np.random.default_rng(n)
    return _molecule(rng.uniform(-1.0, 1.0, (n, 3)) * np.array([4.0, 4.0, 2.0 + n / 8.0]), n + 100)


@pytest.mark.parametrize("family", ["dna", "pydock", "vdw", "cpydock"])
@pytest.mark.parametrize("group", [4, 8, 16, 32])
@pytest.mark.parametrize("n", [1, 3, 4, 5, 17, 33, 130])
def test_lists_match_oracle(family, group, n):
    rec, lig = _dense_receptor(), _ligand(n)
    poses = np.vstack([random_poses(10, [0, 0, 0], 14.0, n), random_poses(6, [24, 0, 0], 6.0, n + 1),
                       random_poses(2, [400, 0, 0], 1.0, n + 2)])
    ref, rparts = oracle.Model(family, rec, lig).batch_energy_grid(poses, parts=True)
    ctx = lkg.Context(group=group)
    cid = ctx.add_complex(family, rec, lig)
    got, parts = ctx.score(cid, poses, parts=True)
    assert np.array_equal(parts[:, 3], rparts[:, 4])
    tol = 1e-6 * (3.0 * parts[:, 3] + np.abs(parts[:, 1])) + 1e-9
    assert np.all(np.abs(got - ref) <= tol)
    assert np.array_equal(got, ctx.score(cid, poses))   # near pairs counted or not, the same bits
    ctx.close()


@pytest.mark.parametrize("tile,group", [(64, 8), (128, 8), (128, 4), (256, 16), (256, 32)])
@pytest.mark.parametrize("n", [3, 65, 300])
def test_split_tiles_score_the_same_bits(tile, group, n):
    # a launch of few poses is split into units of one to a few groups, a
    # large one works in whole tiles: a pose's bits must not depend on it
    rec, lig = _dense_receptor(), _ligand(n)
    poses = random_poses(5, [0, 0, 0], 14.0, n)
    ctx = lkg.Context(tile=tile, group=group)
    cid = ctx.add_complex("dna", rec, lig)
    alone = [ctx.score(cid, p, parts=True) for p in poses]
    for count in (5, 300, 3000, 40000):
        got, parts = ctx.score(cid, np.tile(poses, (count // 5, 1)), parts=True)
        assert np.array_equal(got.reshape(-1, 5), np.tile([a[0][0] for a in alone], (count // 5, 1)))
        assert np.array_equal(parts[:5], np.vstack([a[1] for a in alone]))
    ctx.close()
