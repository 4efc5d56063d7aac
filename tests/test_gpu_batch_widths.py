"""The batch kernel's DP widths of 18, 22, 26 and 30 words per lane, at both ends of the
model lengths of each, at 8, 16 and 32 lanes, against the oracle."""
import numpy as np
import pytest

from cudahmmsearch_gb300 import api
from cudahmmsearch_gb300 import formats as F
from oracle import oracle as O

pytestmark = pytest.mark.gpu
WORDS = [17, 18, 21, 22, 25, 26, 29, 30]


@pytest.mark.parametrize("lanes,lo,hi", [(8, 16, 479), (16, 480, 1023), (32, 1024, 2047)])
def test_widths_match_oracle(lanes, lo, hi):
    ctx = api.Context(0)
    Ms = sorted({M for w in WORDS for M in (2 * lanes * (w - 1), 2 * lanes * w - 1) if lo <= M <= hi} | {lo, hi})
    profs = [api.sample_profile(M, 60 + i, ctx) for i, M in enumerate(Ms)]
    s = F.SeqSet.concat([F.synth_sequences(250, seed=lanes, lmax=4000), F.emit_homologs(profs[0], 15, seed=1),
                         F.emit_homologs(profs[-1], 15, seed=2, repeat=9),
                         F.SeqSet.from_list([np.zeros(0, np.uint8), np.array([3], np.uint8)])])
    xj, fl = api.search_batch(ctx, profs, api.DeviceDB(ctx, s))
    ne = s.lengths > 0
    for i, p in enumerate(profs):
        o = O.msv_batch(p, s)
        ok = o["status"] == F.eslOK
        assert np.array_equal(xj[i][ok], o["xj"][ok]), Ms[i]
        assert np.array_equal((fl[i] & api.FLAG_ERANGE) != 0, o["status"] == F.eslERANGE), Ms[i]
        assert np.array_equal(((fl[i] & api.FLAG_PASS) != 0)[ne], o["pass"][ne] == 1), Ms[i]
        assert np.array_equal(((fl[i] & api.FLAG_FULL) != 0)[ne], o["path"][ne] == 1), Ms[i]
    ctx.close()
