"""Paths of the warp kernels that only some sizes and modes take: the f64 mode at
every group size, ragged quads and refilled lists; a pose's bits with the f64
mode or restraints, alone and in batches; host calls around the size where the
results are copied instead of written by the kernels; cpydock ligands of more
groups than are listed at a time.

Tolerances: the f64 mode's 1e-11 (relative, denominator max(|E|, 1)); in the fast
mode 1e-6 per pair term, as in the candidate lists' own test.
"""
import numpy as np
import pytest

import oracle
from tests.lkg_helpers import lkg, random_poses, rel_err

pytestmark = pytest.mark.gpu


def _mol(coords, seed):
    rng = np.random.default_rng(seed)
    n = len(coords)
    return dict(coords=np.asarray(coords, np.float32).astype(np.float64), ele=rng.uniform(-0.8, 0.8, n),
                vdw=rng.uniform(0.015, 0.25, n), radius=rng.uniform(0.6, 2.1, n),
                heavy=rng.integers(0, 2, n).astype(np.uint8), hyd=rng.integers(0, 2, n).astype(np.int32),
                des=rng.uniform(-0.1, 0.1, n), asa=rng.uniform(-1.0, 70.0, n))


def _receptor():
    g = np.arange(-8, 9) * 2.15   # 17^3 atoms, 0.1 per cubic A
    p = np.stack(np.meshgrid(g, g, g, indexing="ij"), -1).reshape(-1, 3)
    return _mol(p + np.random.default_rng(1).uniform(-0.3, 0.3, p.shape), 2)


def _ligand(n):
    rng = np.random.default_rng(n)
    return _mol(rng.uniform(-1.0, 1.0, (n, 3)) * np.array([4.0, 4.0, 2.0 + n / 8.0]), n + 100)


def _restrain(ctx, cid, rec, lig):
    nr, nl = len(rec["coords"]), len(lig["coords"])
    rr = np.where(np.arange(nr) % 9 == 0, np.arange(nr) // 9 % 50, -1).astype(np.int32)
    lr = np.where(np.arange(nl) % 5 == 0, np.arange(nl) // 5 % 3, -1).astype(np.int32)
    ctx.set_restraints(cid, rr, lr if lr.max() >= 0 else None, np.arange(3, nr, 17, dtype=np.int32))


@pytest.mark.parametrize("family", ["dna", "pydock", "vdw"])
@pytest.mark.parametrize("group", [4, 16, 32])
@pytest.mark.parametrize("n", [1, 5, 33, 130])
def test_f64_lists_match_oracle(family, group, n):
    rec, lig = _receptor(), _ligand(n)
    poses = np.vstack([random_poses(10, [0, 0, 0], 14.0, n), random_poses(6, [24, 0, 0], 6.0, n + 1)])
    ref, rparts = oracle.Model(family, rec, lig).batch_energy_grid(poses, parts=True)
    ctx = lkg.Context(precision="exact", group=group)
    cid = ctx.add_complex(family, rec, lig)
    got, parts = ctx.score(cid, poses, parts=True)
    assert np.array_equal(parts[:, 3], rparts[:, 4])
    assert np.all(rel_err(got, ref) <= 1e-11)
    assert np.array_equal(got, ctx.score(cid, poses))
    ctx.close()


@pytest.mark.parametrize("precision,restrained", [("exact", False), ("exact", True), ("fast", True)])
@pytest.mark.parametrize("tile,group", [(64, 8), (128, 4), (256, 32)])
def test_split_tiles_score_the_same_bits(precision, restrained, tile, group):
    rec, lig = _receptor(), _ligand(300)
    poses = random_poses(5, [0, 0, 0], 14.0, 7)
    ctx = lkg.Context(precision=precision, tile=tile, group=group)
    cid = ctx.add_complex("dna", rec, lig)
    if restrained:
        _restrain(ctx, cid, rec, lig)
    alone = np.array([ctx.score(cid, p)[0] for p in poses])
    for count in (5, 300, 3000):
        got = ctx.score(cid, np.tile(poses, (count // 5, 1)))
        assert np.array_equal(got.reshape(-1, 5), np.tile(alone, (count // 5, 1)))
    ctx.close()


@pytest.mark.parametrize("family,precision", [("vdw", "fast"), ("cpydock", "fast"), ("dna", "exact")])
def test_results_written_or_copied(family, precision):
    rec, lig = _mol(np.random.default_rng(5).uniform(-8.0, 8.0, (300, 3)), 6), _ligand(20)
    poses = random_poses(5000, [9, 0, 0], 6.0, 8)
    ctx = lkg.Context(precision=precision)
    cid = ctx.add_complex(family, rec, lig)
    _restrain(ctx, cid, rec, lig)
    whole, frac = ctx.score_interface(cid, poses)
    assert (frac > 0).any(axis=0).all()
    for count in (1, 16, 17, 4095, 4096, 4097):
        got, f = ctx.score_interface(cid, poses[:count])
        assert np.array_equal(got, whole[:count]) and np.array_equal(f, frac[:count])
        got, parts = ctx.score(cid, poses[:count], parts=True)
        assert np.array_equal(got, whole[:count])
        assert np.array_equal(parts, ctx.score(cid, poses, parts=True)[1][:count])
    ctx.close()


@pytest.mark.parametrize("restrained", [False, True])
@pytest.mark.parametrize("n", [4096, 4097, 4500, 9000])
def test_cpydock_ligands_of_many_groups(n, restrained):
    # groups of 4: 1024 groups are listed at a time
    rng = np.random.default_rng(n)
    rec = _mol(rng.uniform(-9.0, 9.0, (500, 3)), 3)
    lig = _mol(rng.uniform(-1.0, 1.0, (n, 3)) * np.array([60.0, 12.0, 12.0]), 4)
    # the receptor beside every part of the ligand in turn
    along = np.array([[1.0, 0, 0, 0, x, 9.0, 9.0] for x in (-62.0, -40.0, -13.0, 13.0, 40.0, 62.0, 300.0)])
    poses = np.vstack([random_poses(4, [0, 0, 0], 14.0, 5), along])
    m = oracle.Model("cpydock", rec, lig)
    ref, rparts = m.batch_energy_grid(poses, parts=True)
    ctx = lkg.Context(group=4)
    cid = ctx.add_complex("cpydock", rec, lig)
    got, parts = ctx.score(cid, poses, parts=True)
    assert np.array_equal(parts[:, 3], rparts[:, 4])
    assert np.all(np.abs(got - ref) <= 1e-6 * (3.0 * parts[:, 3] + np.abs(parts[:, 1])) + 1e-9)
    if restrained:
        _restrain(ctx, cid, rec, lig)
        s, f = ctx.score_interface(cid, poses)
        ctx16 = lkg.Context(group=16)
        c16 = ctx16.add_complex("cpydock", rec, lig)
        _restrain(ctx16, c16, rec, lig)
        s16, f16 = ctx16.score_interface(c16, poses)
        ctx16.close()
        assert (f > 0).any() and np.array_equal(f, f16)
        assert np.all(rel_err(s, s16) <= 1e-5)
    ctx.close()
