"""Which ViterbiFilter kernel a profile and a database's longest target take
(msvgb_vprofile_packed), and the packed kernel's 8-warp forms on models with
the entry costs of their length, on both sides of the target length it reaches,
against the oracle. Results are integers and their float score: equality."""
import math

import numpy as np
import pytest

from cudahmmsearch_gb300 import api
from cudahmmsearch_gb300 import formats as F
from tests.test_gpu_vit_packed import check, general, homologs, resized, targets, vprofile
from tests.vprofiles import crop_vprofile

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    c = api.Context(0)
    yield c
    c.close()


def scaled(vp, M):
    """resized, with entry costs that fall with the length as a local model's do, and the D->D bound that
    vf_conversion (src/impl_sse/p7_oprofile.c:653-760) sets for them: it rises by as much."""
    v = resized(vp, M)
    k = np.arange(M)
    tw = v.twv.copy()
    fall = round(vp.scale_w * (math.log(M * (M + 1.0)) - math.log(vp.M * (vp.M + 1.0))))
    tw[k % v.Q8 * 7, k // v.Q8] -= np.int16(fall)
    return F.VProfile(M, tw, v.rwv, v.xw, v.scale_w, v.nj, v.base_w, v.ddbound_w + fall)


def reach(dv):
    """The longest target the packed kernel takes (the rule is monotone in the length)."""
    lo, hi = 0, 1 << 26
    while lo < hi:
        mid = (lo + hi + 1) // 2
        lo, hi = (mid, hi) if dv.packed(mid) else (lo, mid - 1)
    return lo


@pytest.mark.parametrize("name,lo,hi", [("m50_s1", 1 << 26, 1 << 26), ("m400_s1", 2_500_000, 2_700_000),
                                        ("m1500_s2", 140_000, 155_000), ("m2400_s1", 42_000, 46_000),
                                        ("vitwide_m4000_s7", 14_000, 15_500)])
def test_reach_of_the_models(ctx, name, lo, hi):
    assert lo <= reach(api.DeviceVProfile(ctx, vprofile(name))) <= hi


@pytest.mark.parametrize("how", ["no_match_path", "no_entry", "dd_bound", "n_loop", "j_loop", "e_loop", "padding"])
def test_refused(ctx, how):
    vp = crop_vprofile(vprofile("m2400_s1"), 150)
    assert api.DeviceVProfile(ctx, vp).packed(1500)
    assert not api.DeviceVProfile(ctx, general(vp, how)).packed(0)


def test_longest_target_decides(ctx):
    dv = api.DeviceVProfile(ctx, crop_vprofile(vprofile("m2400_s1"), 2390))
    assert dv.packed(3000) and not dv.packed(60000)


@pytest.mark.parametrize("M", [4097, 5120, 6200, 8191, 8192])
def test_wide_models_on_both_sides_of_the_reach(ctx, M):
    vp = scaled(vprofile("m2400_s1"), M)
    dv = api.DeviceVProfile(ctx, vp)
    L = reach(dv)
    assert 3000 < L < 20_000 and dv.packed(1500)
    check(ctx, vp, targets(vp, M))
    rng = np.random.default_rng(M)
    for longest in (L, L + 1):                            # packed, general
        s = [rng.integers(0, 20, longest).astype(np.uint8)] + homologs(vp, rng, 10)
        check(ctx, vp, F.SeqSet.from_list(s))


def test_a_real_wide_model(ctx):
    vp = vprofile("vitwide_m4000_s7")
    rng = np.random.default_rng(2)
    for longest in (14_000, 16_000):                      # packed, general
        assert api.DeviceVProfile(ctx, vp).packed(longest) == (longest == 14_000)
        s = [rng.integers(0, 20, longest).astype(np.uint8)] + homologs(vp, rng, 20)
        check(ctx, vp, F.SeqSet.from_list(s))
