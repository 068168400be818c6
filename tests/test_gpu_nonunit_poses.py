"""Quaternions are used as given, without normalisation (as the reference): one of
another length than 1 stretches the ligand across its axis, and the groups'
bounding spheres with it.  Near-pair counts and scores against the oracle, with
the tolerances of the candidate lists' own test (fast) and of the f64 mode.
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


@pytest.mark.parametrize("precision", ["exact", "fast"])
@pytest.mark.parametrize("family,group", [("vdw", 4), ("vdw", 8), ("vdw", 32), ("cpydock", 4), ("cpydock", 8)])
@pytest.mark.parametrize("length", [0.6, 0.97, 1.0005, 1.04, 1.6])
def test_quaternions_of_any_length(precision, family, group, length):
    g = np.arange(-6, 7) * 2.6
    rec = np.stack(np.meshgrid(g, g, g, indexing="ij"), -1).reshape(-1, 3)
    rec = _mol(rec + np.random.default_rng(1).uniform(-0.4, 0.4, rec.shape), 2)
    lig = _mol(np.random.default_rng(3).uniform(-9.0, 9.0, (90, 3)), 4)
    poses = np.vstack([random_poses(12, [0, 0, 0], 14.0, 5), random_poses(20, [26, 0, 0], 6.0, 6)])
    poses[:, :4] *= length
    ctx = lkg.Context(precision=precision, group=group)
    got, parts = ctx.score(ctx.add_complex(family, rec, lig), poses, parts=True)
    ctx.close()
    ref, rparts = oracle.Model(family, rec, lig).batch_energy_grid(poses, parts=True)
    assert np.array_equal(parts[:, 3], rparts[:, 4])
    if precision == "exact":
        assert np.all(rel_err(got, ref) <= 1e-11)
    else:
        assert np.all(np.abs(got - ref) <= 1e-6 * (3.0 * parts[:, 3] + np.abs(parts[:, 1])) + 1e-9)
