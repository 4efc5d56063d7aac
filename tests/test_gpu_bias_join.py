"""Both ends of the bias filter's speculation, shown by a float simulation of the
segments' start states: sequences whose segments join bit for bit, and sequences
that have to be scored from their start. Scores against the oracle: equality."""
import numpy as np
import pytest

from cudahmmsearch_gb300 import api
from cudahmmsearch_gb300 import formats as F
from oracle import oracle as O
from tests.test_gpu_bias_segments import composition

pytestmark = pytest.mark.gpu
SEG, WARM = 512, 1024
f32 = np.float32


def joins(compo, M, seq):
    """Whether every segment's run-in from the guess ends in the state the segment before ends in. Canonical residues."""
    bg = F.AMINO_BG.astype(f32)
    eo = np.stack([bg / bg, compo.astype(f32) / bg], 1)[seq]
    L = len(seq)
    l1 = f32(M / 8.0)
    t10, t11 = f32(1) / (l1 + f32(1)), l1 / (l1 + f32(1))
    t00 = f32(L) / f32(L + 1)
    t01 = f32(1) - t00
    ks = np.arange(3, (L + SEG - 1) // SEG)               # the first three start at the sequence's own first row
    state = {}
    for k in range(2, (L + SEG - 1) // SEG):
        start = k * SEG - WARM
        d0, d1 = f32(1), f32(0.05)
        for i in range(start, min(L, (k + 1) * SEG)):
            if i == 0:
                n0, n1 = eo[0, 0] * f32(0.999), eo[0, 1] * f32(0.001)
            else:
                n0 = (d0 * t00 + d1 * t10) * eo[i, 0]
                n1 = (d0 * t01 + d1 * t11) * eo[i, 1]
            m = max(n0, n1)
            d0, d1 = n0 / m, n1 / m
            if i + 1 == k * SEG:
                state[k, "first"] = (d0, d1)
        state[k, "last"] = (d0, d1)
    return all(state[k, "first"] == state[k - 1, "last"] for k in ks)


def near_background():
    """Odds near 1 for every residue: a long model forgets a state over thousands of rows."""
    bg = F.AMINO_BG.astype(np.float64) / F.AMINO_BG.sum()
    return (bg * (1 + np.random.default_rng(1).normal(0, 1e-3, 20))).astype(f32)


@pytest.mark.parametrize("kind,M,want", [("near", 2000, False), ("near", 8000, False), ("near", 260, True), ("peaked", 260, True)])
def test_joined_and_rescored(kind, M, want):
    rng = np.random.default_rng(M)
    compo = near_background() if kind == "near" else composition(kind)
    seqs = [rng.integers(0, 20, L).astype(np.uint8) for L in (1800, 2049, 2560, 3500, 6000)]
    seen = [joins(compo, M, q) for q in seqs if len(q) > 2 * SEG + WARM]
    assert seen and all(j == want for j in seen)
    s = F.SeqSet.from_list(seqs)
    ctx = api.Context(0)
    got = api.biasfilter(ctx, compo, M, api.DeviceDB(ctx, s))
    assert np.array_equal(got.view(np.uint32), O.bias_batch(compo, M, s).view(np.uint32))
    ctx.close()
