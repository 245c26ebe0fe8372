"""Scratch memory and results of the block-resident decoder with long windows (few lanes of a warp in use:
the compact scratch slot), alone and beside short blocks of the same call.

Bar of the posteriors: the one of test_gpu_resident_range.py, derived there."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import awgn_blocks
from test_gpu_std3gpp import std_code_blocks

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ks,window", [([6144] * 600, 6144), ([6144] * 300 + [40] * 3000, 6144), ([6144] * 1200, 1024)])
def test_scratch_is_sized_by_the_lanes_in_use(tc, ks, window):
    """X of a warp holds 6144 steps, at 16 float4 per 8 steps 197 KB of slot; at most 8 CTAs on each SM and a
    quarter more when the buffer grows: below 300 MB, however long the windows are."""
    import torch

    dec = tc.Decoder(0)
    ks = np.asarray(ks)
    _, llr = dec.awgn_code_blocks_device(5, ks, np.full(ks.size, 1.0, np.float32))
    cbs, llr_len, post_len = tc.Decoder.layout(ks)
    post = torch.zeros(post_len, device="cuda")
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    dec.decode_device(cbs, ks.size, llr.data_ptr(), llr_len, post.data_ptr(), post_len, 0, 0,
                      tc.DecodeOptions(2, False, window))
    torch.cuda.synchronize()
    taken = before - torch.cuda.mem_get_info()[0]
    dec.close()
    assert taken < 320e6, taken


CASES = [
    # blocks, window, guard, early stop, Eb/N0 (4: the (m, s) pass too)
    ([6144, 6144, 40, 48, 512, 1056], 6144, 96, False, 1.0),      # the full trellis
    ([6144] * 3 + [2048] * 5 + [40] * 70, 1024, 96, True, 1.0),   # 6, 2 and 1 windows a block
    ([6144, 4096, 6080], 512, 0, False, 1.0),                     # 12 lanes, no guard, a ragged last window
    ([6144, 5056] * 4, 2048, 2048, False, 4.0),                   # guard = window
    ([3136] * 6 + [104] * 9, 384, 96, True, 4.0),
]


@pytest.mark.parametrize("std", [False, True])
@pytest.mark.parametrize("ks,window,guard,early,ebn0", CASES)
def test_long_windows(tc, decoder, oracle, ks, window, guard, early, ebn0, std):
    if std:
        llr = std_code_blocks(tc, ks, ebn0, 41)[0]
    else:
        llr = awgn_blocks(tc, ks, ebn0, 41, crc24b=early)[0]
    conv = tc.CONVENTION_3GPP if std else tc.CONVENTION_REFERENCE
    post, ok, used = decoder.decode(ks, llr, None, tc.DecodeOptions(6, early, window, guard, convention=conv))
    one = oracle.std_decode_cb if std else oracle.decode_cb
    lo = po = 0
    for i, k in enumerate(ks):
        ref, rok, rused = one(k, 0, llr[lo:lo + 3 * (k + 4)], 6, early, window=min(window, k), guard=guard)
        ref = ref.astype(np.float64)
        bar = np.maximum(1e-3 * np.maximum(np.abs(ref), 1.0), 2e-5 * np.abs(ref).max())
        assert (bool(ok[i]), int(used[i])) == (rok, rused), (i, k)
        assert (np.abs(post[po:po + k] - ref) <= bar).all(), (i, k)
        lo += 3 * (k + 4)
        po += k
