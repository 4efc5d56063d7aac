"""Searches that cut their long targets into segments (and skip blocks of the
full MSV by the segments' largest cells), and the 4-lane passes of short
models, against the oracle: model lengths on every kernel width family, targets
from one row to many segments, homologs inside long targets (undecided after
SSV, some overflowing), SSV disabled by length, repeated searches on one
context. Results are integers: equality, no tolerance."""
import os

import numpy as np
import pytest

from cudahmmsearch_gb300 import api
from cudahmmsearch_gb300 import formats as F
from oracle import oracle as O

pytestmark = pytest.mark.gpu
GOLDEN = os.path.join(os.path.dirname(__file__), "golden")


@pytest.fixture(scope="module")
def ctx():
    c = api.Context(0)
    yield c
    c.close()


def planted(p, seed, lengths, copies):
    """Background sequences of the given lengths, with weakened copies of the
    model's best residues planted in two thirds of them."""
    rng = np.random.default_rng(seed)
    best = p.node_costs()[:20].argmin(0)
    bg = np.cumsum(F.AMINO_BG.astype(np.float64) / F.AMINO_BG.sum())
    out = []
    for i, L in enumerate(lengths):
        s = np.minimum(np.searchsorted(bg, rng.random(L)), 19).astype(np.uint8)
        for _ in range(copies if i % 3 else 0):
            n = int(min(L, rng.integers(4, max(5, min(p.M, 150)))))
            k, at = int(rng.integers(0, p.M - n + 1)) if p.M > n else 0, int(rng.integers(0, L - n + 1))
            n = min(n, p.M - k)
            core = best[k:k + n].copy()
            noise = rng.random(n) < rng.choice([0.1, 0.4, 0.6, 0.7])
            core[noise] = rng.integers(0, 20, int(noise.sum()))
            s[at:at + n] = core
        out.append(s)
    return F.SeqSet.from_list(out)


def check(p, s, xj, fl, idx=None):
    idx = np.arange(s.n) if idx is None else idx
    o = O.msv_batch(p, s.subset(idx))
    gx, gf = xj[idx], fl[idx]
    some = s.lengths[idx] > 0
    ok = (o["status"] == 0) & some
    assert np.array_equal((gf & api.FLAG_ERANGE) != 0, o["status"] == 16)
    assert np.array_equal(gx[ok], o["xj"][ok])
    assert np.array_equal(((gf & api.FLAG_PASS) != 0)[some], o["pass"][some] == 1)
    return o


LENGTHS = [0, 1, 17, 300, 511, 512, 513, 1023, 1024, 1025, 1537, 2047, 2600, 4095, 4096, 5000, 9001, 17000, 33000]


@pytest.mark.parametrize("M", [1, 9, 40, 63, 127, 200, 255, 256, 300, 511, 640, 1023, 1100, 1500, 2047, 2100, 2600, 4200])
def test_small_search_with_long_targets(ctx, M):
    p = api.sample_profile(M, M + 1, ctx)
    s = F.SeqSet.concat([planted(p, M, LENGTHS * 2, 3), F.synth_sequences(200, seed=M, lmax=900)])
    dp, db = api.DeviceProfile(ctx, p), api.DeviceDB(ctx, s)
    xj, fl = api.search(ctx, dp, db)
    check(p, s, xj, fl)
    again = api.search(ctx, dp, db)                       # the counts start from zero again
    assert np.array_equal(again[0], xj) and np.array_equal(again[1], fl)
    host = api.search_host(ctx, dp, s)
    assert np.array_equal(host[0], xj) and np.array_equal(host[1], fl)


@pytest.mark.parametrize("M,n", [(20, 200_000), (60, 120_000), (127, 60_000), (200, 60_000), (255, 60_000), (450, 60_000),
                                 (900, 40_000), (1300, 30_000)])
def test_large_search_with_long_targets(ctx, M, n):
    """The lane-group passes (4 lanes for the short models): the whole database
    against the 32-lane kernel, the long targets and a sample against the oracle."""
    p = api.sample_profile(M, M, ctx)
    s = F.SeqSet.concat([planted(p, M, LENGTHS * 8 + [20000] * 8, 4), F.synth_sequences(n, seed=M, lmax=8000)])
    dp, db = api.DeviceProfile(ctx, p), api.DeviceDB(ctx, s)
    xj, fl = api.search(ctx, dp, db)
    d32 = api.DeviceProfile(ctx, p)
    d32.set_lanes(32)
    x32, f32 = api.search(ctx, d32, db)
    assert np.array_equal(xj, x32)
    assert np.array_equal(fl & 0x0b, f32 & 0x0b)          # all flags but "the full MSV ran"
    check(p, s, xj, fl, np.concatenate([np.arange(170), np.random.default_rng(M).choice(s.n, 500, replace=False)]))
    host = api.search_host(ctx, dp, s)
    assert np.array_equal(host[0], xj) and np.array_equal(host[1], fl)
    bx, bf = api.search_batch(ctx, [p, p], db)
    assert np.array_equal(bx[0], xj) and np.array_equal(bx[1], xj) and np.array_equal(bf[0] & 0x0b, fl & 0x0b)


@pytest.mark.parametrize("bias,tbm,base", [(14, 120, 190), (40, 100, 190), (90, 130, 190), (60, 40, 255), (14, 20, 100)])
@pytest.mark.parametrize("M", [150, 700, 2100])
def test_extreme_costs(ctx, M, bias, tbm, base):
    """SSV disabled for long targets, begin scores clamped, base below the move costs."""
    rng = np.random.default_rng(M + bias)
    costs = np.minimum(255, rng.integers(0, 80, size=(F.KP_AMINO, M))).astype(np.uint8)
    p = F.profile_from_node_costs(costs, tbm_b=tbm, tec_b=3, base_b=base, bias_b=bias, scale_b=3.0 / 0.6931471805599453,
                                  mmu=-9.0, mlambda=0.69)
    s = F.SeqSet.concat([planted(p, M, LENGTHS, 2), F.synth_sequences(100, seed=M, lmax=3000)])
    xj, fl = api.search(ctx, api.DeviceProfile(ctx, p), api.DeviceDB(ctx, s))
    check(p, s, xj, fl)


@pytest.mark.parametrize("M", [9, 200, 1500])
def test_dropin_long_targets(ctx, M):
    """The drop-in shares one long target over its block's warps."""
    p = api.sample_profile(M, M + 3)
    s = planted(p, M, [1, 2, 15, 100, 300, 1000, 3000, 7999, 8000, 30000, 301, 2999], 2)
    o = O.msv_batch(p, s)
    for i in range(s.n):
        L = int(s.lengths[i])
        dsq = np.concatenate([[255], s.seq(i), [255]]).astype(np.uint8)
        st, sc = ctx.MSVFilter(dsq, L, p, api.tjb_b(p.scale_b, L))
        assert st == o["status"][i]
        if st == 0:
            assert np.float32(sc).view(np.uint32) == o["sc"][i].view(np.uint32)


def test_words_set_by_hand(ctx):
    """8-bit words set on a profile that chose its lanes itself."""
    p = api.sample_profile(200, 5, ctx)
    s = F.SeqSet.concat([planted(p, 1, LENGTHS, 3), F.synth_sequences(60_000, seed=3, lmax=4000)])
    db = api.DeviceDB(ctx, s)
    dp = api.DeviceProfile(ctx, p)
    assert dp.lanes == 8 and dp.int8_words == 4
    want = api.search(ctx, dp, db)
    dp.set_int8_words(0)
    got = api.search(ctx, dp, db)
    assert dp.int8_words == 0
    assert np.array_equal(got[0], want[0]) and np.array_equal(got[1] & 0x0b, want[1] & 0x0b)
