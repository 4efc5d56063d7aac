"""The route of a resident search by its launches: the fused kernel (one launch)
below the residues that the model's width sets, the lane groups (a pass and its
list) above, on both sides of each line; a sample of every search against the
oracle. Results are integers: equality."""
import numpy as np
import pytest

from cudahmmsearch_gb300 import api
from cudahmmsearch_gb300 import formats as F
from tests.test_gpu_segments import check

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    c = api.Context(0)
    yield c
    c.close()


_SEQS = {}


def of_residues(millions):
    """A prefix of one set of sequences with about this many million residues."""
    if not _SEQS:
        _SEQS["all"] = F.synth_sequences(200_000, seed=5, lmax=12_000)
    s = _SEQS["all"]
    n = int(np.searchsorted(s.off, millions * 1e6)) - 1
    return F.SeqSet(s.codes[:s.off[n]], s.off[:n + 1])


@pytest.mark.parametrize("M,below,above", [(86, 22, 26), (255, 22, 26), (256, 34, 38), (300, 38, 42), (319, 34, 38), (350, 22, 26), (384, 34, 38),
                                           (447, 34, 38), (448, 56, 64), (511, 56, 64), (576, 56, 64), (767, 56, 64),
                                           (768, 40, 44), (1023, 40, 44), (1030, 56, 64), (1090, 40, 44), (1900, 40, 44)])
def test_both_sides_of_the_line(ctx, M, below, above):
    p = api.sample_profile(M, M, ctx)
    dp = api.DeviceProfile(ctx, p)
    for millions, fused in ((below, True), (above, False)):
        s = of_residues(millions)
        db = api.DeviceDB(ctx, s)
        before = api.kernel_launches()
        xj, fl = api.search(ctx, dp, db)
        assert (api.kernel_launches() - before == 1) == fused
        check(p, s, xj, fl, np.random.default_rng(M).choice(s.n, 200, replace=False))
        db.close()
    dp.close()
