"""The surrogate's 16 anchor atoms do not depend on how the scoring kernels order
atoms inside a group: they are sampled farthest point first from the ligand's
bisection into groups.  With a single unit charge as receptor the potential at
an anchor is 1 / d^2, so the features tell which atoms the anchors are.

Tolerance: bf16 features (2^-9), trilinear interpolation of 1 / d^2 on the 0.5 A
grid at 15 A and more (h^2 / 8 * 6 / d^2 * 3 axes < 0.3 %): 1 %; anchors are
several A apart, which changes 1 / d^2 by more.
"""
import numpy as np
import pytest
import torch

from tests.lkg_helpers import lkg

pytestmark = pytest.mark.gpu


def _bisect(c, idx, size):
    if len(idx) <= size:
        return list(idx)
    ax = int(np.argmax(c[idx].max(0) - c[idx].min(0)))
    idx = np.array(sorted(idx, key=lambda i: (c[i, ax], i)))
    left = ((len(idx) + size - 1) // size) // 2 * size
    return _bisect(c, idx[:left], size) + _bisect(c, idx[left:], size)


def _anchors(c, size):
    p = np.asarray(c, np.float32)[_bisect(c, np.arange(len(c)), size)]
    dmin, cur, out = np.full(len(p), 1e30, np.float32), 0, []
    for _ in range(16):
        out.append(p[cur])
        dmin = np.minimum(dmin, ((p - p[cur]) ** 2).sum(1))
        cur = int(np.argmax(dmin))
    return np.array(out, np.float64)


@pytest.mark.parametrize("group,n", [(4, 40), (8, 150), (16, 333), (32, 70)])
def test_anchors_follow_the_group_order(group, n):
    rng = np.random.default_rng(n)
    lig = rng.uniform(-5.0, 5.0, (n, 3)).astype(np.float32).astype(np.float64)
    one = dict(coords=np.zeros((1, 3)), ele=np.ones(1), vdw=np.full(1, 0.1), radius=np.ones(1))
    mol = dict(coords=lig, ele=np.zeros(n), vdw=np.full(n, 0.1), radius=np.ones(n))
    ctx = lkg.Context(group=group)
    sur = lkg.Surrogate(ctx, ctx.add_complex("pydock", one, mol))
    poses = np.array([[1, 0, 0, 0, 21, 0, 0], [1, 0, 0, 0, 0, 21, 0], [1, 0, 0, 0, 0, 0, 21]], float)
    ctx.score(0, poses)
    d = torch.from_numpy(poses).cuda()
    torch.cuda.synchronize()
    f = torch.from_numpy(sur.features_device(3, d.data_ptr()).view(np.int16)).view(torch.bfloat16).double().numpy()
    for k in range(3):
        want = 100.0 / ((_anchors(lig, group) + poses[k, 4:]) ** 2).sum(1)
        assert np.all(np.abs(f[k, 7:7 + 48:3] - want) <= 0.01 * want)
    sur.close()
    ctx.close()
