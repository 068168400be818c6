"""A ligand atom without a finite position is near nothing, and the atoms of its
group keep their own pairs (as in the oracle, which takes atom by atom).

Tolerances: those of the candidate lists' own test (fast) and of the f64 mode.
"""
import numpy as np
import pytest

import oracle
from tests.lkg_helpers import lkg, random_poses, rel_err

pytestmark = pytest.mark.gpu


def _mol(n, size, seed):
    rng = np.random.default_rng(seed)
    return dict(coords=rng.uniform(-size, size, (n, 3)), ele=rng.uniform(-0.5, 0.5, n), vdw=rng.uniform(0.02, 0.2, n),
                radius=rng.uniform(1.0, 2.0, n), heavy=rng.integers(0, 2, n).astype(np.uint8),
                hyd=np.ones(n, np.int32), des=rng.uniform(-0.1, 0.1, n), asa=rng.uniform(1.0, 60.0, n))


@pytest.mark.parametrize("value", [np.nan, np.inf, -np.inf])
@pytest.mark.parametrize("precision", ["exact", "fast"])
@pytest.mark.parametrize("family,group", [("vdw", 4), ("vdw", 8), ("vdw", 32), ("cpydock", 8)])
def test_the_other_atoms_keep_their_pairs(precision, family, group, value):
    rec, lig = _mol(900, 14.0, 1), _mol(50, 6.0, 2)
    lig["coords"][[0, 21]] = value
    lig["coords"][40, 1] = value
    poses = random_poses(12, [4, 0, 0], 10.0, 3)
    ctx = lkg.Context(precision=precision, group=group)
    got, parts = ctx.score(ctx.add_complex(family, rec, lig), poses, parts=True)
    ctx.close()
    ref, rparts = oracle.Model(family, rec, lig).batch_energy_grid(poses, parts=True)
    assert rparts[:, 4].min() > 0
    assert np.array_equal(parts[:, 3], rparts[:, 4])
    if family == "cpydock":   # the desolvation sum of an atom that is nowhere is not defined
        return
    if precision == "exact":
        assert np.all(rel_err(got, ref) <= 1e-11)
    else:
        assert np.all(np.abs(got - ref) <= 1e-6 * (3.0 * parts[:, 3] + np.abs(parts[:, 1])) + 1e-9)
