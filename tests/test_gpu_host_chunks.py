"""The route of a host search in several chunks, by its launches: the fused kernel
where a chunk is too small to fill the lane groups, the groups for short models,
large databases and databases of mostly long targets. Results equal the resident
search's."""
import numpy as np
import pytest

from cudahmmsearch_gb300 import api
from cudahmmsearch_gb300 import formats as F

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    c = api.Context(0)
    yield c
    c.close()


@pytest.fixture(scope="module")
def databases():
    short = F.synth_sequences(200_000, seed=3, lmax=2000)
    assert 64 << 20 < short.total < 90e6                  # several chunks
    rng = np.random.default_rng(1)
    long = F.SeqSet.from_list([rng.integers(0, 20, 8000).astype(np.uint8) for _ in range(9000)])
    return {"short": short, "long": long}


@pytest.mark.parametrize("M,targets,groups", [(20, "short", True), (200, "short", False), (420, "short", False),
                                              (900, "short", True), (200, "long", True)])
def test_route(ctx, databases, M, targets, groups):
    """A pack and one pass per chunk are an even count; the groups add one list for all."""
    s = databases[targets]
    p = api.sample_profile(M, M, ctx)
    dp, db = api.DeviceProfile(ctx, p), api.DeviceDB(ctx, s)
    before = api.kernel_launches()
    xj, fl = api.search_host(ctx, dp, s)
    assert ((api.kernel_launches() - before) % 2 == 1) == groups
    rx, rf = api.search(ctx, dp, db)
    assert np.array_equal(xj, rx) and np.array_equal(fl & 0x0b, rf & 0x0b)
    db.close()
