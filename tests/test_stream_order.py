"""What a kernel on a context's stream reads next is written on that stream.  The
streams are created non-blocking, and a cudaMemcpy from pageable memory or a
cudaMemset may return before the device memory holds its last bytes: a kernel
launched next could read the old contents.
"""
import os
import re

import numpy as np
import pytest

from tests.lkg_helpers import REPO, lkg, random_poses

CSRC = os.path.join(REPO, "lklight-gpu_b200", "csrc")


@pytest.mark.parametrize("name", sorted(f for f in os.listdir(CSRC) if f.endswith((".cu", ".cpp", ".cuh", ".h"))))
def test_no_upload_or_clear_outside_a_stream(name):
    with open(os.path.join(CSRC, name)) as f:
        src = re.sub(r"//[^\n]*", "", f.read())
    calls = re.findall(r"\bcuda(?:Memcpy|Memset|MemcpyToSymbol)\s*\([^;]*;", src)
    assert [c for c in calls if "cudaMemcpyDeviceToHost" not in c] == []


@pytest.mark.gpu
@pytest.mark.parametrize("family", ["dna", "cpydock"])
def test_restraint_tags_set_moved_and_cleared(family):
    # a receptor of 4 kB of flags, the tags changed before every call: each call
    # equals that of a context which only ever had these tags
    rng = np.random.default_rng(4)

    def mol(n, size):
        return dict(coords=rng.uniform(-size, size, (n, 3)), ele=rng.uniform(-0.5, 0.5, n),
                    vdw=rng.uniform(0.02, 0.2, n), radius=rng.uniform(1.0, 2.0, n),
                    heavy=np.ones(n, np.uint8), hyd=np.ones(n, np.int32), des=rng.uniform(-0.1, 0.1, n),
                    asa=rng.uniform(0.0, 60.0, n))

    rec, lig = mol(256, 12.0), mol(40, 5.0)
    poses = random_poses(6, [12, 0, 0], 4.0, 9)
    tags = []
    for k in range(3):
        rr = np.full(256, -1, np.int32)
        rr[k::7] = np.arange(len(rr[k::7])) % 4
        tags.append((rr, np.arange(k, 256, 11, dtype=np.int32)))
    want = []
    for rr, mem in tags + [(None, None)]:
        ctx = lkg.Context()
        cid = ctx.add_complex(family, rec, lig)
        if rr is not None:
            ctx.set_restraints(cid, rr, None, mem)
        want.append(ctx.score_interface(cid, poses))
        ctx.close()
    assert any((w[1] > 0).any() for w in want[:3])
    ctx = lkg.Context()
    cid = ctx.add_complex(family, rec, lig)
    for turn in range(60):
        k = turn % 4
        if k < 3:
            ctx.set_restraints(cid, tags[k][0], None, tags[k][1])
        else:
            ctx.set_restraints(cid)
        got = ctx.score_interface(cid, poses)
        assert np.array_equal(got[0], want[k][0]) and np.array_equal(got[1], want[k][1])
    ctx.close()
