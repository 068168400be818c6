"""cpydock complexes of a default context: ligands of up to 700 atoms are searched by
groups of 8, larger ones by 16, each size in a launch of its own.  Mixed batches
around the line, against the oracle and against each complex alone.

Tolerance: that of the candidate lists' own test (1e-6 per pair term).
"""
import numpy as np
import pytest

import oracle
from tests.lkg_helpers import lkg, random_poses

pytestmark = pytest.mark.gpu


def _mol(n, box, seed):
    rng = np.random.default_rng(seed)
    return dict(coords=rng.uniform(-1.0, 1.0, (n, 3)) * np.asarray(box), ele=rng.uniform(-0.8, 0.8, n),
                vdw=rng.uniform(0.015, 0.25, n), radius=rng.uniform(0.6, 2.1, n),
                heavy=rng.integers(0, 2, n).astype(np.uint8), hyd=rng.integers(0, 2, n).astype(np.int32),
                des=rng.uniform(-0.1, 0.1, n), asa=rng.uniform(-1.0, 70.0, n))


@pytest.mark.parametrize("precision", ["fast", "exact"])
def test_ligands_around_the_line_in_one_batch(precision):
    rec = [_mol(n, (12.0, 12.0, 12.0), n) for n in (700, 300)]
    items = [("cpydock", rec[0], _mol(n, (9.0, 9.0, 3.0 + n / 60.0), n)) for n in (1, 9, 17, 130, 699, 700, 701, 720)]
    items += [("dna", rec[1], _mol(40, (6.0, 6.0, 6.0), 5)), ("cpydock", rec[1], _mol(5, (3.0, 3.0, 3.0), 6))]
    poses = [random_poses(6 + k, [10, 0, 0], 9.0, k) for k in range(len(items))]
    ctx = lkg.Context(precision=precision)
    ids = [ctx.add_complex(*it) for it in items]
    counts = [len(p) for p in poses]
    alone = [ctx.score(i, p, parts=True) for i, p in zip(ids, poses)]
    got = np.zeros(sum(counts))
    parts = np.zeros((sum(counts), 4))
    ctx.score_multi(ids, counts, np.vstack(poses), got, parts)
    assert np.array_equal(got, np.concatenate([a[0] for a in alone]))
    assert np.array_equal(parts, np.vstack([a[1] for a in alone]))
    for (family, r, l), p, (s, q) in zip(items, poses, alone):
        ref, rparts = oracle.Model(family, r, l).batch_energy_grid(p, parts=True)
        assert np.array_equal(q[:, 3], rparts[:, 4])
        assert np.all(np.abs(s - ref) <= 1e-6 * (3.0 * q[:, 3] + np.abs(q[:, 1])) + 1e-9)
    ctx.close()
