"""Searches that cut no target: the 32-lane kernel for whole sequences
(msvgb_search_static, both tables) at the edges of its widths, eight rows a step
over targets of every remainder; the lane-group passes and their list without
segments (lanes set by hand, with the default and with other 8-bit words).
Results are integers: equality."""
import ctypes

import numpy as np
import pytest

from cudahmmsearch_gb300 import api
from cudahmmsearch_gb300 import formats as F
from tests.test_gpu_segments import check, planted

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
SHORT = [0, 1, 2, 3, 4, 5, 7, 8, 9, 15, 16, 17, 23, 24, 25, 31, 32, 33, 300, 301, 999, 1000, 3001]


@pytest.fixture(scope="module")
def ctx():
    c = api.Context(0)
    yield c
    c.close()


def static(ctx, dp, db):
    out = torch.full((2, db.n), 99, dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    st = api.lib().msvgb_search_static(dp.h, db.h, 0.02, ctypes.c_void_p(out[0].data_ptr()),
                                       ctypes.c_void_p(out[1].data_ptr()), None)
    assert st == api.eslOK
    torch.cuda.synchronize()
    return out[0].cpu().numpy(), out[1].cpu().numpy()


@pytest.mark.parametrize("M", [1, 63, 64, 127, 130, 191, 192, 319, 447, 511, 512, 703, 1023, 1024, 1087, 1340, 1535, 2047, 2048,
                               2300, 2559, 2560, 3000, 4100, 5000, 6200, 7300, 8191])
def test_f16_widths(ctx, M):
    p = api.sample_profile(M, M + 1, ctx)
    s = F.SeqSet.concat([planted(p, M, SHORT * 3, 2), F.synth_sequences(60, seed=M, lmax=900)])
    check(p, s, *static(ctx, api.DeviceProfile(ctx, p), api.DeviceDB(ctx, s)))


@pytest.mark.parametrize("M", [1, 127, 128, 255, 600, 1500, 2300, 3100])
def test_int8_widths(ctx, M):
    p = api.sample_profile(M, M + 1, ctx)
    s = F.SeqSet.concat([planted(p, M, SHORT * 3, 2), F.synth_sequences(60, seed=M, lmax=900)])
    dp = api.DeviceProfile(ctx, p, variant=0)
    assert dp.variant == 0
    check(p, s, *static(ctx, dp, api.DeviceDB(ctx, s)))


@pytest.mark.parametrize("G,M", [(8, 16), (8, 95), (8, 160), (8, 303), (8, 368), (8, 448), (8, 511), (16, 40), (16, 300), (16, 415),
                                 (16, 607), (16, 736), (16, 880), (16, 1023), (32, 1100), (32, 1470), (32, 1790), (32, 2047)])
def test_lanes_by_hand(ctx, G, M):
    p = api.sample_profile(M, M + 2, ctx)
    s = F.SeqSet.concat([planted(p, M, SHORT * 3 + [2399, 2400, 5000, 9001], 3), F.synth_sequences(300, seed=M, lmax=2000)])
    db, dp = api.DeviceDB(ctx, s), api.DeviceProfile(ctx, p)
    dp.set_lanes(G)
    check(p, s, *api.search(ctx, dp, db))
    if G < 32 and dp.int8_words:
        dp.set_int8_words(0)
        check(p, s, *api.search(ctx, dp, db))
