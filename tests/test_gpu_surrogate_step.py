"""A surrogate training step at the sizes where its launches change: one row, the
edges of the 32-row partial sums and of the 128-row tiles, and the batch size
at which the weight gradients and backward products stop sharing launches; and
long trainings (replayed from a graph) against short ones (launched one by one).

Tolerances as in test_gpu_surrogate.py: 1e-2 on the outputs, 3 % relative L2 per
gradient block against the oracle with the device's BF16 rounding points.
"""
import numpy as np
import pytest
import torch

from oracle import mlp as omlp
from tests.lkg_helpers import lkg, random_poses

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx_cid():
    rng = np.random.default_rng(8)

    def mol(n, spread):
        return dict(coords=rng.uniform(-spread, spread, (n, 3)), ele=rng.uniform(-0.5, 0.5, n),
                    vdw=np.full(n, 0.1), radius=np.full(n, 1.5))
    ctx = lkg.Context()
    yield ctx, ctx.add_complex("pydock", mol(900, 14.0), mol(120, 6.0))
    ctx.close()


@pytest.mark.parametrize("n", [1, 31, 33, 127, 129, 1024, 9472, 9473])
def test_gradient_at_launch_edges(ctx_cid, n):
    sur = lkg.Surrogate(*ctx_cid, seed=1)
    rng = np.random.default_rng(n)
    p = omlp.he_params(n).astype(np.float32)
    sur.set_params(p)
    X = omlp.f64_to_bf16_bits(rng.normal(0.0, 1.0, size=(n, omlp.IN)))
    t = rng.normal(0.0, 1.0, n).astype(np.float32)
    y, g, loss = sur.grad(X, t)
    l_ref, g_ref, y_ref = omlp.loss_and_grad(p.astype(np.float64), omlp.bf16_bits_to_f64(X), t.astype(np.float64),
                                             emulate=True)
    assert np.abs(y - y_ref).max() < 1e-2 * (1.0 + np.abs(y_ref).max())
    assert abs(loss - l_ref) < 1e-2 * (1.0 + l_ref)
    o = 0
    for size in omlp.SIZES:
        a, b = g[o:o + size].astype(np.float64), g_ref[o:o + size]
        assert np.linalg.norm(a - b) <= 3e-2 * max(np.linalg.norm(b), 1e-12)
        o += size
    assert sur.status() == 0
    sur.close()


def test_graph_and_plain_launches_train_the_same_bits(ctx_cid):
    ctx, cid = ctx_cid
    poses = random_poses(700, [0, 0, 0], 18.0, 4)
    known = ctx.score(cid, poses)
    d, k = torch.from_numpy(poses).cuda(), torch.from_numpy(known).cuda()
    torch.cuda.synchronize()
    out = []
    for parts in ((32,), (8, 8, 16), (1,) * 32):
        sur = lkg.Surrogate(ctx, cid, seed=3)
        sur.set_target_scale(known)
        for e in parts:
            loss = sur.train_device(len(poses), d.data_ptr(), k.data_ptr(), epochs=e, batch=256)
        out.append((sur.params(), loss))
        sur.close()
    for p, loss in out[1:]:
        assert np.array_equal(p, out[0][0]) and loss == out[0][1]
