"""Searches captured into a CUDA graph on the context's stream: a later search
with a larger need of segment scratch leaves the graph's buffers alone, and a
search whose scratch would have to grow is captured all the same (its long
targets then run uncut). Results are integers: equality, no tolerance."""
import numpy as np
import pytest

from cudahmmsearch_gb300 import api
from cudahmmsearch_gb300 import formats as F
from oracle import oracle as O

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def random_targets(seed, counts):
    rng = np.random.default_rng(seed)
    return F.SeqSet.from_list([rng.integers(0, 20, L).astype(np.uint8) for L, n in counts for _ in range(n)])


class Captured:
    """A search into its own result buffers, captured on its own stream."""

    def __init__(self, ctx, dp, db):
        self.out = torch.full((2, db.n), 99, dtype=torch.uint8, device="cuda")
        self.stream, self.graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
        torch.cuda.synchronize()
        ctx.set_stream(self.stream.cuda_stream)
        with torch.cuda.graph(self.graph, stream=self.stream):
            api.search_device(ctx, dp, db, self.out[0].data_ptr(), self.out[1].data_ptr())
        ctx.set_stream(None)

    def run(self):
        self.out.fill_(99)
        torch.cuda.synchronize()
        self.graph.replay()
        torch.cuda.synchronize()
        return self.out.cpu().numpy()


def equal_oracle(p, s, xj, fl):
    o = O.msv_batch(p, s)
    ok = o["status"] == 0
    return (np.array_equal(xj[ok], o["xj"][ok]) and np.array_equal((fl & api.FLAG_ERANGE) != 0, o["status"] == 16)
            and np.array_equal((fl & api.FLAG_PASS) != 0, o["pass"] == 1))


def test_replay_after_a_search_with_a_larger_need():
    ctx = api.Context(0)
    s = random_targets(1, [(300, 20_000), (9000, 8), (33_000, 2)])
    db = api.DeviceDB(ctx, s)
    wide, narrow = api.sample_profile(2000, 3, ctx), api.sample_profile(60, 4, ctx)
    dw, dn = api.DeviceProfile(ctx, wide), api.DeviceProfile(ctx, narrow)
    api.search(ctx, dw, db)                               # the need of a wide model: its ten long targets only
    g = Captured(ctx, dw, db)
    xj, fl = api.search(ctx, dn, db)                      # every target is long for a short model
    out = g.run()
    assert equal_oracle(wide, s, out[0], out[1])
    assert equal_oracle(narrow, s, xj, fl)
    again = api.search(ctx, dn, db)
    assert np.array_equal(again[0], xj) and np.array_equal(again[1], fl)
    ctx.close()


def test_capture_does_not_grow_the_scratch():
    ctx = api.Context(0)
    p = api.sample_profile(60, 5, ctx)
    dp = api.DeviceProfile(ctx, p)
    few = api.DeviceDB(ctx, random_targets(2, [(200, 30_000), (300, 10), (33_000, 4)]))
    s = random_targets(3, [(300, 20_000), (33_000, 4)])
    db = api.DeviceDB(ctx, s)
    api.search(ctx, dp, few)                              # the lengths' tables and the list; little scratch
    g = Captured(ctx, dp, db)
    out = g.run()
    assert equal_oracle(p, s, out[0], out[1])
    xj, fl = api.search(ctx, dp, db)                      # cut, outside the capture
    assert np.array_equal(xj, out[0]) and np.array_equal(fl & 0x0b, out[1] & 0x0b)
    ctx.close()
