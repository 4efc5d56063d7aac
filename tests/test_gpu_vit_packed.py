"""The packed ViterbiFilter kernel (two nodes per register, fused add-maximum)
and the rule that sends a profile to it, against the oracle: model lengths at
the edges of its row widths, rows it scores with saturation (large scores,
gap and other non-residue codes), profiles and targets the rule must leave to
the general kernels, and both kernels on the same inputs. Results are integers
and their float score: equality, no tolerance."""
import os

import numpy as np
import pytest

from cudahmmsearch_gb300 import api
from cudahmmsearch_gb300 import formats as F
from oracle import oracle as O
from tests.vprofiles import crop_vprofile

pytestmark = pytest.mark.gpu
GOLDEN = os.path.join(os.path.dirname(__file__), "golden")


@pytest.fixture(scope="module")
def ctx():
    c = api.Context(0)
    yield c
    c.close()


def vprofile(name):
    return F.read_vprofile(os.path.join(GOLDEN, "vit_" + name + ".vprof"))


def homologs(vp, rng, n):
    """Sequences following the model's best residues, with noise (scores from small to saturating)."""
    k = np.arange(vp.M)
    best = vp.rwv[:20, k % vp.Q8, k // vp.Q8].argmax(0)
    out = []
    for i in range(n):
        a = int(rng.integers(0, max(1, vp.M - 5)))
        core = best[a:a + int(rng.integers(3, 120))].copy()
        noise = rng.random(core.size) < i / n
        core[noise] = rng.integers(0, 20, int(noise.sum()))
        out.append(np.concatenate([rng.integers(0, 20, int(rng.integers(0, 40))), core]).astype(np.uint8))
    return out


def targets(vp, seed):
    rng = np.random.default_rng(seed)
    s = [rng.integers(0, 20, L).astype(np.uint8) for L in (1, 2, 3, 4, 5, 15, 16, 17, 33, 400, 1500)]
    s += homologs(vp, rng, 40)
    for L in (1, 5, 60, 300):                             # every code, gaps and non-residues among them
        s.append(rng.integers(0, 29, L).astype(np.uint8))
        s.append(np.full(L, 20 if L % 2 else 27, np.uint8))
    for t in homologs(vp, rng, 20):                       # a non-residue inside a strong match
        t[int(rng.integers(0, t.size))] = rng.choice([20, 27, 28])
        s.append(t)
    s.append(np.zeros(0, np.uint8))
    return F.SeqSet.from_list(s)


def check(ctx, vp, s):
    o = O.vit_batch(vp, s)
    st, sc = api.vitfilter(ctx, api.DeviceVProfile(ctx, vp), api.DeviceDB(ctx, s))
    want = np.where(s.lengths == 0, 2, np.where(o["status"] == 16, 1, 0))
    assert np.array_equal(st, want)
    ok = want == 0
    assert np.array_equal(sc[ok].view(np.uint32), o["sc"][ok].view(np.uint32))
    return st


def resized(vp, M):
    """A profile of M nodes: cropped, or its inner nodes repeated."""
    if M <= vp.M:
        return crop_vprofile(vp, M)
    k = np.arange(M)
    src = np.where(k == 0, 0, 1 + (k - 1) % (vp.M - 2))
    Q0, Q8 = vp.Q8, (M - 1) // 8 + 1
    tw = np.full((8 * Q8, 8), -32768, np.int16)
    rw = np.full((vp.Kp, Q8, 8), -32768, np.int16)
    for t in range(7):
        tw[k % Q8 * 7 + t, k // Q8] = vp.twv[src % Q0 * 7 + t, src // Q0]
    tw[7 * Q8 + k % Q8, k // Q8] = vp.twv[7 * Q0 + src % Q0, src // Q0]
    for t in (4, 5, 6):
        tw[(M - 1) % Q8 * 7 + t, (M - 1) // Q8] = -32768
    tw[7 * Q8 + (M - 1) % Q8, (M - 1) // Q8] = -32768
    rw[:, k % Q8, k // Q8] = vp.rwv[:, src % Q0, src // Q0]
    return F.VProfile(M, tw, rw, vp.xw, vp.scale_w, vp.nj, vp.base_w, vp.ddbound_w)


@pytest.mark.parametrize("M", [1, 2, 5, 63, 64, 65, 127, 128, 129, 511, 512, 513, 896, 897, 1024, 1025, 1280, 1281,
                               2303, 2304, 2399, 3072, 3584, 3585, 4096, 4097, 5120, 6200, 8191, 8192])
def test_row_widths(ctx, M):
    vp = resized(vprofile("m2400_s1"), M)
    check(ctx, vp, targets(vp, M))


@pytest.mark.parametrize("name", ["tut_fn3", "tut_globins4", "tut_pkinase", "m33_s3", "m777_s3", "m1500_s2"])
def test_models(ctx, name):
    vp = vprofile(name)
    st = check(ctx, vp, targets(vp, vp.M))
    assert (st == 1).any() or vp.M < 40                   # some targets overflow


def general(vp, how):
    """A copy the packed kernel's rule must refuse: the general kernels score it."""
    tw, rw, xw, dd = vp.twv.copy(), vp.rwv.copy(), np.array(vp.xw), vp.ddbound_w
    Q8, k = vp.Q8, vp.M // 2                              # node k, 0-based
    if how == "no_match_path":
        tw[k % Q8 * 7 + 1, k // Q8] = -32768
    elif how == "no_entry":
        tw[k % Q8 * 7, k // Q8] = -32768
    elif how == "dd_bound":
        dd = -32768
    elif how == "n_loop":
        xw[1][1] = -3
    elif how == "j_loop":
        xw[2][1] = -3
    elif how == "e_loop":
        xw[0][1] = 40
    elif how == "padding":
        rw[3, vp.M % Q8, vp.M // Q8] = 100
    return F.VProfile(vp.M, tw, rw, xw, vp.scale_w, vp.nj, vp.base_w, dd)


@pytest.mark.parametrize("how", ["no_match_path", "no_entry", "dd_bound", "n_loop", "j_loop", "e_loop", "padding"])
@pytest.mark.parametrize("M", [61, 150, 1276])
def test_refused_profiles(ctx, M, how):
    vp = general(crop_vprofile(vprofile("m2400_s1"), M), how)
    check(ctx, vp, targets(vp, M))


@pytest.mark.parametrize("how", ["match", "emission", "dd"])
@pytest.mark.parametrize("cost", [-14000, -20000, -26000])
def test_low_costs(ctx, how, cost):
    """Costs on either side of what the rule accepts, at one node."""
    vp = crop_vprofile(vprofile("m400_s1"), 180)
    tw, rw, Q8, k = vp.twv.copy(), vp.rwv.copy(), vp.Q8, 70
    if how == "match":
        tw[k % Q8 * 7 + 1, k // Q8] = cost
    elif how == "emission":
        rw[5, k % Q8, k // Q8] = cost
    else:
        tw[7 * Q8 + k % Q8, k // Q8] = cost
    low = F.VProfile(vp.M, tw, rw, vp.xw, vp.scale_w, vp.nj, vp.base_w, vp.ddbound_w)
    check(ctx, low, targets(low, -cost))


def test_long_targets(ctx):
    """The rule holds up to a target length; a database with longer ones runs on the general kernel."""
    vp = crop_vprofile(vprofile("m2400_s1"), 2390)
    rng = np.random.default_rng(5)
    for L in (3000, 60000):
        s = F.SeqSet.from_list([rng.integers(0, 20, L).astype(np.uint8)] + homologs(vp, rng, 10))
        check(ctx, vp, s)


def test_both_kernels_agree(ctx):
    """The same scores from both kernels on a survivor list: an entry cost the
    rule refuses at a node no path can use (every way into it closed)."""
    vp = vprofile("tut_pkinase")
    Q8, k = vp.Q8, vp.M - 1                               # the last node
    tw, rw = vp.twv.copy(), vp.rwv.copy()
    rw[:, k % Q8, k // Q8] = -32768
    a = F.VProfile(vp.M, tw, rw, vp.xw, vp.scale_w, vp.nj, vp.base_w, vp.ddbound_w)
    tw = tw.copy()
    tw[k % Q8 * 7, k // Q8] = -32768
    b = F.VProfile(vp.M, tw, rw, vp.xw, vp.scale_w, vp.nj, vp.base_w, vp.ddbound_w)
    s = F.SeqSet.concat([F.synth_sequences(2000, seed=9, lmax=3000), targets(vp, 3)])
    db = api.DeviceDB(ctx, s)
    ids = np.arange(s.n - 1, -1, -3)
    ra, rb = (api.vitfilter(ctx, api.DeviceVProfile(ctx, v), db, ids) for v in (a, b))
    assert np.array_equal(ra[0], rb[0]) and np.array_equal(ra[1].view(np.uint32), rb[1].view(np.uint32))
