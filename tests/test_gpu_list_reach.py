"""The candidate lists hold every pair within the cutoff, however large the
coordinates and the ligand's groups are: near-pair counts equal the oracle's.
Positions are tested against the spheres of groups and quads in f32, whose
rounding grows with the coordinates (0.008 A at 1e5 A) and with the square of a
group's width.

Tolerance of the scores in the f64 mode: at 1e5 A a coordinate's last place is
1.5e-11 A, which moves a term by at most 14 x 1.5e-11 relative at 1 A: 1e-9.
"""
import numpy as np
import pytest

import oracle
from tests.lkg_helpers import lkg, rel_err

pytestmark = pytest.mark.gpu


def _mol(coords, seed):
    rng = np.random.default_rng(seed)
    n = len(coords)
    return dict(coords=np.asarray(coords, float), ele=rng.uniform(-0.8, 0.8, n), vdw=rng.uniform(0.015, 0.25, n),
                radius=rng.uniform(0.6, 2.1, n), heavy=rng.integers(0, 2, n).astype(np.uint8))


def _score(precision, group, family, rec, lig, poses):
    ctx = lkg.Context(precision=precision, group=group)
    got, parts = ctx.score(ctx.add_complex(family, rec, lig), poses, parts=True)
    ctx.close()
    ref, rparts = oracle.Model(family, rec, lig).batch_energy_grid(poses, parts=True)
    return got, parts[:, 3], ref, rparts[:, 4]


def _shells(step, width, seed):
    # 16 clumps of 4 atoms in a row, each in a shell of receptor atoms whose
    # distances lie around the cutoff: a pair is at the very edge of its quad's sphere
    rng = np.random.default_rng(seed)
    centre = (np.arange(16) - 7.5)[:, None] * np.array([step, 0.0, 0.0])
    lig = np.repeat(centre, 4, 0) + rng.uniform(-0.2, 0.2, (64, 3)) * width
    u = rng.normal(size=(16 * 60, 3))
    u /= np.linalg.norm(u, axis=1, keepdims=True)
    rec = np.repeat(centre, 60, 0) + u * (10.0 + width * rng.uniform(-1.0, 1.0, (16 * 60, 1)))
    poses = np.hstack([np.tile([1.0, 0.0, 0.0, 0.0], (40, 1)), 0.3 * width * rng.uniform(-1.0, 1.0, (40, 3))])
    return rec, lig, poses


# (the fast mode holds the receptor in f32: up to some 480 A the rounding of a
# distance stays inside the band around the cutoff that f64 decides)
@pytest.mark.parametrize("precision,step", [("exact", 3.0), ("exact", 40.0), ("exact", 1000.0), ("fast", 3.0),
                                            ("fast", 40.0)])
@pytest.mark.parametrize("group", [4, 8, 16, 32])
def test_groups_of_any_width(precision, group, step):
    rec, lig, poses = _shells(step, 0.02, int(step))
    got, near, ref, rnear = _score(precision, group, "vdw", _mol(rec, 1), _mol(lig, 2), poses)
    assert rnear.min() > 100
    assert np.array_equal(near, rnear)
    tol = 1e-9 if precision == "exact" else 1e-6 * (3.0 * near + np.abs(ref))   # as the lists' own test
    assert np.all(np.abs(got - ref) <= tol * np.maximum(np.abs(ref), 1.0))


@pytest.mark.parametrize("frame", ["receptor", "ligand"])
@pytest.mark.parametrize("group", [4, 8, 32])
@pytest.mark.parametrize("far", [1e3, 1e5, -1e6])
def test_coordinates_of_any_size(frame, group, far):
    rec, lig, poses = _shells(12.0, 0.02 + 1e-7 * abs(far), 7)
    at = far * np.array([1.0, -0.7, 0.4])
    if frame == "receptor":
        rec = rec + at
        poses[:, 4:7] += at
    else:
        lig = lig + at
        poses[:, 4:7] -= at
    got, near, ref, rnear = _score("exact", group, "vdw", _mol(rec, 1), _mol(lig, 2), poses)
    assert rnear.min() > 100
    assert np.array_equal(near, rnear)
    # (a coordinate's last place grows with its size)
    assert np.all(rel_err(got, ref) <= 1e-9 * max(1.0, abs(far) / 1e5))
