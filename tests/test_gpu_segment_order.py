"""The fused kernel's last segment to finish runs the full MSV from block maxima
that other warps and CTAs wrote: many long targets whose segments end at nearly
the same time, each skipping rows by those maxima, scored again and again and
against the oracle. A stale maximum would skip a row that raises the score.
Results are integers: equality, no tolerance."""
import numpy as np
import pytest

from cudahmmsearch_gb300 import api
from cudahmmsearch_gb300 import formats as F
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def weak_matches(p, seed, lengths, copies):
    """Random sequences with short, noisy stretches of the model's best residues: enough for the full MSV,
    too few to overflow it."""
    rng = np.random.default_rng(seed)
    best = p.node_costs()[:20].argmin(0)
    out = []
    for L in lengths:
        s = rng.integers(0, 20, L).astype(np.uint8)
        for _ in range(copies):
            n = int(rng.integers(4, 8))
            k, at = int(rng.integers(0, p.M - n + 1)), int(rng.integers(0, L - n + 1))
            core = best[k:k + n].copy()
            noise = rng.random(n) < 0.4
            core[noise] = rng.integers(0, 20, int(noise.sum()))
            s[at:at + n] = core
        out.append(s)
    return F.SeqSet.from_list(out)


@pytest.mark.parametrize("M", [130, 200, 700])
def test_last_segment_reads_every_block(M):
    ctx = api.Context(0)
    p = api.sample_profile(M, M + 7, ctx)
    s = weak_matches(p, M, [3000 + 37 * i for i in range(300)], 6)
    o = O.msv_batch(p, s)
    ok = o["status"] == 0
    assert ((o["path"] == 1) & ok).mean() > 0.3           # undecided after SSV: the full MSV reads the maxima
    dp, db = api.DeviceProfile(ctx, p), api.DeviceDB(ctx, s)
    for _ in range(20):
        xj, fl = api.search(ctx, dp, db)
        assert np.array_equal((fl & api.FLAG_ERANGE) != 0, o["status"] == 16)
        assert np.array_equal(xj[ok], o["xj"][ok])
    ctx.close()
