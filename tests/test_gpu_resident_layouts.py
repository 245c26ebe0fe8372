"""The layouts of the block-resident decoder, each shown to run there (one launch per decode; a launch per
half-iteration and three more otherwise): CTAs of 32, 64, 96 and 128 threads, several blocks per CTA, windows
from 8 steps on, windows that do not divide the block, guard 0 and guard = window, both codes; and the calls
that keep a launch per half-iteration.  Against the oracle running the same windows.

Bar of the posteriors: 1e-4 max(|ref| of the block, 1), as in test_gpu_resident.py, derived there."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import awgn_blocks
from test_gpu_std3gpp import std_code_blocks

pytestmark = pytest.mark.gpu


def _window(k, persistent, target, guard):
    """The window that a block of size k is cut into (decoder.cu, decode_now)."""
    if not persistent:
        return min(target, k)
    nwin = max(1, min(32, k // max(target, 8)))
    wlen = -(-(-(-k // nwin)) // 8) * 8
    if nwin > 1 and wlen < guard:
        nwin = max(1, k // guard)
        wlen = -(-(-(-k // nwin)) // 8) * 8
    return min(wlen, k)


def _check(tc, decoder, oracle, ks, persistent, window, guard, early, std, iters, launches):
    llr = std_code_blocks(tc, ks, 1.0, 51)[0] if std else awgn_blocks(tc, ks, 1.0, 51, crc24b=early)[0]
    decoder.timing(reset=True)
    post, ok, used = decoder.decode(ks, llr, None, tc.DecodeOptions(
        iters, early, window, guard, tc.SCHEDULE_PERSISTENT if persistent else tc.SCHEDULE_PLAIN,
        convention=tc.CONVENTION_3GPP if std else tc.CONVENTION_REFERENCE))
    assert decoder.timing()["launches"] == launches
    one = oracle.std_decode_cb if std else oracle.decode_cb
    lo = po = 0
    for i, k in enumerate(ks):
        if len(ks) < 50 or i < 3 or i + 3 >= len(ks) or i % 37 == 0:
            ref, rok, rused = one(k, 0, llr[lo:lo + 3 * (k + 4)], iters, early,
                                  window=_window(k, persistent, window, guard), guard=guard)
            err = np.abs(post[po:po + k].astype(np.float64) - ref).max()
            assert err <= 1e-4 * max(np.abs(ref).max(), 1.0), (i, k, err)
            assert (bool(ok[i]), int(used[i])) == (rok, rused), (i, k)
        lo += 3 * (k + 4)
        po += k


RESIDENT = [
    # blocks, persistent schedule, window, guard, early stop
    ([40], False, 128, 96, False),                            # one window of 40 steps
    ([40, 48, 64, 512, 1056, 40], True, 8, 8, True),          # windows of 8 steps on, blocks sharing a warp
    ([1024, 1024, 256], True, 8, 32, False),                  # 32 windows of 32; guard = window
    ([2048, 1504, 40], True, 8, 0, True),                     # no guard, a ragged last window
    ([1056] * 9, True, 64, 64, False),
    ([4096] * 3, False, 128, 96, False),                      # 32 windows: one warp exactly
    ([4160, 40], False, 128, 96, True),                       # 33: 64 threads
    ([6144, 4096], False, 136, 96, True),                     # 64 threads, a ragged last window
    ([6080, 1504], False, 152, 0, False),                     # no guard
    ([6144] * 2, False, 128, 128, False),                     # guard = window
    ([6144] * 300, False, 128, 96, False),                    # two blocks in 96 threads
    ([5120] * 297 + [40] * 50, False, 128, 96, True),         # three in 128, and short ones
    ([5376] * 300, False, 128, 0, False),                     # 42 windows: 126 of 128 threads
]


@pytest.mark.parametrize("std", [False, True])
@pytest.mark.parametrize("ks,persistent,window,guard,early", RESIDENT)
def test_resident(tc, decoder, oracle, ks, persistent, window, guard, early, std):
    _check(tc, decoder, oracle, ks, persistent, window, guard, early, std, 5, 1)


@pytest.mark.parametrize("ks,persistent,window,iters", [
    ([512, 1056], False, 64, 5),       # windows below 128: the differentiable decoder's schedule
    ([6144] * 1200, False, 2048, 2),   # long windows in more than one wave
])
def test_launch_per_half_iteration(tc, decoder, oracle, ks, persistent, window, iters):
    _check(tc, decoder, oracle, ks, persistent, window, 64, False, False, iters, 2 * iters + 3)
