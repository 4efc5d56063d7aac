"""The tuner times each lane choice for the length mix the way a profile with
that choice runs: 16 and 8 lanes with their long targets cut into segments (two
launches a search, not three), 8 lanes below 256 nodes on 4. The launches of a
tuning run are counted against the table it leaves."""
import pytest

from cudahmmsearch_gb300 import api

pytestmark = pytest.mark.gpu
RUNS = 4                                                  # one warm-up and three timed runs of each choice
BINS = 4


def lane_choices(M):
    return sum(2 <= M // (2 * g) + 1 <= 32 for g in (16, 8))


def test_the_mix_is_timed_as_it_runs(tmp_path):
    ctx = api.Context(0)
    before = api.kernel_launches()
    path = str(tmp_path / "table.txt")
    assert ctx.autotune(budget_s=2.0, cache=path) == "measured"
    launches = api.kernel_launches() - before
    Ms = [int(l.split()[1]) for l in open(path) if l.startswith("m ")]
    assert Ms
    want = BINS + 1                                       # the databases
    for M in Ms:
        want += RUNS * (2 + 2 * lane_choices(M))          # the mix: 32 lanes (two tables) fused, the others two passes
        want += RUNS * BINS * (1 + lane_choices(M))       # the bins, one graph a run
    assert launches == want
    ctx.close()
