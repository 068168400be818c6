"""A ligand atom whose desolvation parameter is not finite spoils the score of
every pose in every cpydock kernel (0 x inf is not a number where no receptor
atom is near), as in the oracle: groups out of the receptor's reach included.
"""
import numpy as np
import pytest

import oracle
from tests.lkg_helpers import lkg

pytestmark = pytest.mark.gpu


def _mol(n, size, seed):
    rng = np.random.default_rng(seed)
    return dict(coords=rng.uniform(-size, size, (n, 3)), ele=rng.uniform(-0.5, 0.5, n), vdw=rng.uniform(0.02, 0.2, n),
                radius=rng.uniform(1.0, 2.0, n), heavy=np.ones(n, np.uint8), hyd=np.ones(n, np.int32),
                des=rng.uniform(-0.1, 0.1, n), asa=rng.uniform(1.0, 60.0, n))


@pytest.mark.parametrize("value", [np.inf, -np.inf, np.nan])
@pytest.mark.parametrize("precision,group", [("fast", 4), ("fast", 8), ("fast", 16), ("fast", 32), ("exact", 8)])
def test_far_groups_keep_a_nonfinite_parameter(precision, group, value):
    rec, lig = _mol(400, 10.0, 1), _mol(70, 7.0, 2)
    poses = np.array([[1.0, 0, 0, 0, x, 0, 0] for x in (0.0, 25.0, 40.0, 70.0)])
    ctx = lkg.Context(precision=precision, group=group)
    whole = ctx.score(ctx.add_complex("cpydock", rec, lig), poses)
    assert np.isfinite(whole).all()
    lig["des"][33] = value
    got = ctx.score(ctx.add_complex("cpydock", rec, lig), poses)
    ctx.close()
    ref = oracle.Model("cpydock", rec, lig).batch_energy_grid(poses)
    assert not np.isfinite(ref).any()
    assert np.array_equal(np.isnan(got), np.isnan(ref)) and not np.isfinite(got).any()
