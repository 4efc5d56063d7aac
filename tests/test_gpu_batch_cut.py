"""A batch's own searches (profiles whose search fills the GPU alone) with long
targets cut into many segments inside the captured graph: replayed several
times, on all of its branches, against the plain search and the oracle. Results
are integers: equality, no tolerance."""
import numpy as np
import pytest

from cudahmmsearch_gb300 import api
from cudahmmsearch_gb300 import formats as F
from oracle import oracle as O
from tests.test_gpu_segments import planted

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def test_own_searches_cut_their_targets():
    ctx = api.Context(0)
    Ms = [220, 400, 700, 1100, 1500, 2100]                # 4, 8, 16 and 32 lanes, and the fused kernel
    profs = [api.sample_profile(M, M + 2, ctx) for M in Ms]
    long = planted(profs[1], 3, [35_000, 60_000, 120_000, 200_000] * 3, 4)
    s = F.SeqSet.concat([long, planted(profs[3], 4, [9000] * 20, 3), F.synth_sequences(500_000, seed=5, lmax=3000)])
    assert min(Ms) * s.total >= 40e9                      # every profile's search is its own
    # at 32 lanes a chain scores about this many rows, and so does a segment: the longest targets have several
    assert s.total / (152 * 24) < 100_000
    db = api.DeviceDB(ctx, s)
    out = torch.zeros((2, len(Ms), s.n), dtype=torch.uint8, device="cuda")
    b = api.Batch(ctx, profs, db, out[0].data_ptr(), out[1].data_ptr())
    first = None
    for _ in range(3):
        out.fill_(99)
        torch.cuda.synchronize()
        b.run()
        torch.cuda.synchronize()
        got = out.cpu().numpy()
        assert first is None or np.array_equal(got, first)
        first = got
    idx = np.concatenate([np.arange(long.n + 20), np.random.default_rng(1).choice(s.n, 300, replace=False)])
    for i, p in enumerate(profs):
        xj, fl = api.search(ctx, api.DeviceProfile(ctx, p), db)
        assert np.array_equal(got[0, i], xj), p.M
        assert np.array_equal(got[1, i] & 0x0b, fl & 0x0b), p.M
        o = O.msv_batch(p, s.subset(idx))
        ok = o["status"] == 0
        assert np.array_equal(xj[idx][ok], o["xj"][ok]), p.M
        assert np.array_equal((fl[idx] & api.FLAG_ERANGE) != 0, o["status"] == 16), p.M
        assert np.array_equal((fl[idx] & api.FLAG_PASS) != 0, o["pass"] == 1), p.M
    b.close()
    ctx.close()
