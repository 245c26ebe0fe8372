"""The block-resident decoder where its layout or its arithmetic changes: CTAs of 32 to 256 threads,
several blocks per CTA, windows that do not divide the block, no guard, one long window, layouts
that take a launch per half-iteration instead (more than 256 windows, X beyond shared memory), and
blocks that leave the linear domain at once, after some iterations, or not at all.  Against the
oracle running the same windows, which evaluates the same recursion in float32.

Bar: |gpu - ref| <= 1e-4 max(|ref| of the block, 1).  A step rounds metrics of up to the block's
largest |posterior| R once (2^-24 R), a half-iteration's errors are carried by a window of some 100
steps whose metrics add (as independent roundings: 10 x 2^-24 R) and 12 to 16 half-iterations add up:
about 16 x 10 x 2^-24 = 1e-5 of R, on either side; 1e-4 leaves a factor of 5.
"""
from __future__ import annotations

import numpy as np
import pytest

from conftest import awgn_blocks

pytestmark = pytest.mark.gpu

CASES = [
    # blocks, window, guard, Eb/N0, early stop, iterations, factor on the LLRs
    ([40], 64, 32, 1.0, False, 6, 1.0),                         # one window
    ([40, 48, 64, 512, 1056, 40], 64, 32, 1.0, True, 6, 1.0),   # blocks sharing a warp
    ([2048], 64, 64, 1.0, False, 6, 1.0),                       # 32 windows; guard = window
    ([2112], 64, 32, 1.0, False, 6, 1.0),                       # 33: 64 threads
    ([6144, 40], 64, 32, 1.0, False, 6, 1.0),                   # 96 threads
    ([6144, 4096], 48, 48, 1.0, True, 6, 1.0),                  # 128 threads
    ([6144, 1024], 24, 24, 1.0, False, 6, 1.0),                 # 256 threads, all in use
    ([6080, 1504], 56, 0, 1.0, True, 6, 1.0),                   # ragged last windows, no guard
    ([1024], 8, 8, 1.0, False, 6, 1.0),                         # the shortest windows
    ([6144], 16, 16, 1.0, False, 6, 1.0),                       # 384 windows: launches
    ([6144, 512], 2048, 96, 1.0, False, 6, 1.0),                # long windows
    ([6144] * 40, 128, 96, 3.5, False, 8, 1.0),                 # leaves the linear domain late
    ([512, 6144], 128, 96, 1.0, False, 6, 12.0),                # parities too large from the start
]


@pytest.mark.parametrize("ks,window,guard,ebn0,early,iters,factor", CASES)
def test_against_the_windowed_oracle(tc, decoder, oracle, ks, window, guard, ebn0, early, iters, factor):
    llr, _ = awgn_blocks(tc, ks, ebn0, 7 * window + guard, crc24b=early)
    llr = (factor * llr).astype(np.float32)
    post, ok, used = decoder.decode(ks, llr, None, tc.DecodeOptions(iters, early, window, guard))
    lo = po = 0
    for i, k in enumerate(ks):
        if i < 4 or i + 4 >= len(ks):
            ref, rok, rused = oracle.decode_cb(k, 0, llr[lo:lo + 3 * (k + 4)], iters, early, window=min(window, k),
                                               guard=guard)
            err = np.abs(post[po:po + k].astype(np.float64) - ref).max()
            assert err <= 1e-4 * max(np.abs(ref).max(), 1.0), (i, k, err)
            assert (bool(ok[i]), int(used[i])) == (rok, rused), (i, k)
        lo += 3 * (k + 4)
        po += k
