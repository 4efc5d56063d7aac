"""A database whose block maxima would pass the segment scratch's limit (many
targets long enough to be cut, and one of two million rows): its search must run
as one without segments does, the longest target at 32 lanes beside the
lane-group pass and not in it. Results are integers: equality, no tolerance."""
import numpy as np
import pytest

from cudahmmsearch_gb300 import api
from cudahmmsearch_gb300 import formats as F
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def test_one_huge_target_runs_beside_the_pass():
    ctx = api.Context(0)
    rng = np.random.default_rng(8)
    n, L, huge = 132_000, 512, 1 << 21                    # n * huge / 256 blocks: above a GiB
    codes = rng.integers(0, 20, n * L + huge, dtype=np.uint8)
    s = F.SeqSet(codes, np.concatenate([np.arange(n + 1) * L, [n * L + huge]]).astype(np.int64))
    p = api.sample_profile(86, 6, ctx)
    dp, db = api.DeviceProfile(ctx, p), api.DeviceDB(ctx, s)
    before = api.kernel_launches()
    xj, fl = api.search(ctx, dp, db)
    assert api.kernel_launches() - before == 3            # the long target, the lane-group pass, the list
    idx = np.concatenate([[n], rng.choice(n, 2000, replace=False)])
    o = O.msv_batch(p, s.subset(idx))
    ok = o["status"] == 0
    assert np.array_equal(xj[idx][ok], o["xj"][ok])
    assert np.array_equal((fl[idx] & api.FLAG_ERANGE) != 0, o["status"] == 16)
    assert np.array_equal((fl[idx] & api.FLAG_PASS) != 0, o["pass"] == 1)
    host = api.search_host(ctx, dp, s)
    assert np.array_equal(host[0], xj) and np.array_equal(host[1] & 0x0b, fl & 0x0b)
    ctx.close()
