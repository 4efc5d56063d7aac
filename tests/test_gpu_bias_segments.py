"""The bias filter's segments of long sequences (scored from a guessed state
and joined where the states agree bit for bit) against the oracle: lengths at
the edges of a segment, its run-in and the shortest sequence that is cut;
sequences whose state the guess does not reach; more rows than one call cuts;
a composition that takes both divisions of a row."""
import numpy as np
import pytest

from cudahmmsearch_gb300 import api
from cudahmmsearch_gb300 import formats as F
from oracle import oracle as O

pytestmark = pytest.mark.gpu
EDGES = [k + d for k in (512, 1024, 1536, 2048, 2560, 3072, 4608) for d in (-1, 0, 1, 15, 16, 17)]


@pytest.fixture(scope="module")
def ctx():
    c = api.Context(0)
    yield c
    c.close()


def composition(kind):
    rng = np.random.default_rng(4)
    if kind == "background":                             # forgets a state slowest
        c = np.full(20, 0.05) + rng.normal(0, 1e-4, 20)
    elif kind == "peaked":
        c = rng.dirichlet(np.full(20, 0.3))
    else:                                                # a residue whose odds need both divisions
        c = rng.dirichlet(np.full(20, 2.0))
        c[7] = 1e30
    return c.astype(np.float32)


@pytest.mark.parametrize("kind,M", [("background", 2000), ("background", 30), ("peaked", 260), ("both divisions", 260)])
def test_segments_match_oracle(ctx, kind, M):
    rng = np.random.default_rng(M)
    compo = composition(kind)
    seqs = [rng.integers(0, 20, size=L).astype(np.uint8) for L in EDGES + [9001, 35000]]
    seqs += [np.full(L, x, np.uint8) for L, x in ((4000, 0), (4001, 7), (2049, 26))]          # one residue
    seqs += [np.repeat(rng.integers(0, 20, size=40), 150).astype(np.uint8) for _ in range(10)]  # runs of one
    seqs += [rng.integers(0, 29, size=5000, dtype=np.uint8)]
    s = F.SeqSet.concat([F.SeqSet.from_list(seqs), F.synth_sequences(50, seed=M, lmax=1500)])
    want = O.bias_batch(compo, M, s).view(np.uint32)
    db = api.DeviceDB(ctx, s)
    assert np.array_equal(api.biasfilter(ctx, compo, M, db).view(np.uint32), want)
    ids = rng.integers(0, s.n, size=300)                 # any order, sequences listed more than once
    assert np.array_equal(api.biasfilter(ctx, compo, M, db, ids).view(np.uint32), want[ids])


def test_more_long_sequences_than_one_call_cuts(ctx):
    rng = np.random.default_rng(6)
    compo = composition("peaked")
    s = F.SeqSet.from_list([rng.integers(0, 20, size=int(L)).astype(np.uint8)
                            for L in rng.integers(1400, 6000, size=1600)])
    assert s.total > 4 << 20
    want = O.bias_batch(compo, 300, s)
    assert np.array_equal(api.biasfilter(ctx, compo, 300, api.DeviceDB(ctx, s)).view(np.uint32), want.view(np.uint32))
