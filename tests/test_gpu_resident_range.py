"""The block-resident decoder near the end of its probabilities' range: what it returns there is as exact
as elsewhere, whether a block stayed in the linear form, in its two-factor form, or went on in the (m, s)
form.  Fixed iterations between 2 and 7 dB, where the extrinsics reach 100 to 200 nats, flat and fading
channels, single large parities, evidence that contradicts itself (LLRs of no codeword), both codes, both
schedules, every block against the oracle's 64-bit decoder running the same windows (its float32 decoder is
itself 1.5e-3 off on fading blocks that the iterations do not settle).

Bar: |gpu - ref| <= max(1e-3 max(|ref|, 1), 2e-5 of the block's largest |ref|).  The first is the library's
bar; the second is float32's: a step rounds metrics of up to the block's largest |posterior| R once (2^-24
R), some 100 steps of a window and 16 half-iterations add up as independent roundings: 1e-5 R.
"""
from __future__ import annotations

from concurrent.futures import ThreadPoolExecutor

import numpy as np
import pytest

from conftest import awgn_blocks, schedule_window
from test_gpu_std3gpp import std_code_blocks

pytestmark = pytest.mark.gpu


def _compare(tc, decoder, oracle, ks, llr, iters, persistent=False, std=False, guard=96):
    sched = tc.SCHEDULE_PERSISTENT if persistent else tc.SCHEDULE_PLAIN
    conv = tc.CONVENTION_3GPP if std else tc.CONVENTION_REFERENCE
    post, _, _ = decoder.decode(ks, llr, None, tc.DecodeOptions(iters, False, 0, guard, sched, convention=conv))
    ks = np.asarray(ks, np.int64)
    out = np.concatenate([[0], np.cumsum(ks)])
    at = np.concatenate([[0], np.cumsum(3 * (ks + 4))])

    def worst(i):
        k = int(ks[i])
        ref = oracle.adj_vjp(k, llr[at[i]:at[i + 1]], [1.0] * (2 * iters), schedule_window(k, persistent), guard,
                             std=std)[0]
        bar = np.maximum(1e-3 * np.maximum(np.abs(ref), 1.0), 2e-5 * np.abs(ref).max())
        return float((np.abs(post[out[i]:out[i + 1]] - ref) / bar).max())

    with ThreadPoolExecutor(16) as pool:
        over = np.array(list(pool.map(worst, range(ks.size))))
    bad = np.flatnonzero(~(over <= 1.0))
    assert bad.size == 0, (bad.size, ks.size, int(bad[0]), float(over.max()))


@pytest.mark.parametrize("persistent", [False, True])
@pytest.mark.parametrize("ebn0", [2.5, 2.8, 3.0, 3.2, 4.0])
def test_full_size_blocks(tc, decoder, oracle, ebn0, persistent):
    ks = [6144] * 48
    llr, _ = awgn_blocks(tc, ks, ebn0, 31)
    _compare(tc, decoder, oracle, ks, llr, 8, persistent)


@pytest.mark.parametrize("persistent", [False, True])
@pytest.mark.parametrize("ebn0", [1.5, 2.0, 3.0])
def test_full_size_blocks_of_the_std_code(tc, decoder, oracle, ebn0, persistent):
    ks = [6144] * 32
    llr, _ = std_code_blocks(tc, ks, ebn0, 32)
    _compare(tc, decoder, oracle, ks, llr, 8, persistent, std=True)


@pytest.mark.parametrize("std", [False, True])
@pytest.mark.parametrize("k,n,ebn0", [(40, 4000, 6.0), (40, 4000, 7.0), (512, 300, 4.0), (1056, 200, 3.5)])
def test_short_blocks(tc, decoder, oracle, k, n, ebn0, std):
    ks = [k] * n
    llr = std_code_blocks(tc, ks, ebn0, 33)[0] if std else awgn_blocks(tc, ks, ebn0, 33)[0]
    _compare(tc, decoder, oracle, ks, llr, 8, std=std)


@pytest.mark.parametrize("std", [False, True])
@pytest.mark.parametrize("k,n", [(40, 4000), (512, 200)])
def test_fading(tc, decoder, oracle, k, n, std):
    """Rayleigh fading per code bit at 6 dB: LLRs of very different sizes side by side."""
    rng = np.random.default_rng(34)
    ks = [k] * n
    # noise-free LLRs of size 1 give the code bits
    x = std_code_blocks(tc, ks, 40.0, 34)[0] if std else awgn_blocks(tc, ks, 40.0, 34)[0]
    h = np.sqrt(rng.exponential(size=x.size))
    sigma2 = 1.5 / 10 ** 0.6
    llr = (2 / sigma2 * h * (h * np.sign(x) + np.sqrt(sigma2) * rng.normal(size=x.size))).astype(np.float32)
    _compare(tc, decoder, oracle, ks, llr, 8, std=std)


@pytest.mark.parametrize("std", [False, True])
@pytest.mark.parametrize("value", [-95.0, -60.0, 50.0])
def test_one_large_parity(tc, decoder, oracle, value, std):
    """A single parity LLR of a size of its own among ordinary ones: 2^-137, 2^-87 and 2^72 as weights."""
    ks = [40, 512, 6144] * 16
    llr = std_code_blocks(tc, ks, 1.0, 35)[0] if std else awgn_blocks(tc, ks, 1.0, 35)[0]
    lo = 0
    for i, k in enumerate(ks):
        which = 1 + i % 2
        llr[lo + which * (k + 4) + (k // 2 + i) % k] = value
        lo += 3 * (k + 4)
    _compare(tc, decoder, oracle, ks, llr, 2, std=std)


@pytest.mark.parametrize("std", [False, True])
@pytest.mark.parametrize("k,n,size", [(40, 20000, 40.0), (40, 20000, 50.0), (128, 6000, 40.0), (512, 500, 30.0)])
def test_no_codeword(tc, decoder, oracle, k, n, size, std):
    """Independent uniform LLRs: every step contradicts its neighbours.  One iteration: on noise the
    iterations' own dynamics multiply any rounding."""
    rng = np.random.default_rng(36)
    ks = [k] * n
    llr = rng.uniform(-size, size, n * 3 * (k + 4)).astype(np.float32)
    _compare(tc, decoder, oracle, ks, llr, 1, std=std)


@pytest.mark.parametrize("std", [False, True])
@pytest.mark.parametrize("iters,guard", [(2, 0), (3, 0), (2, 8)])
def test_restart_from_the_beginning(tc, decoder, oracle, iters, guard, std):
    """LLRs three times too large at 1.5 dB: a tenth of the blocks fail their checks all at once at the third
    half-iteration or later and start again.  Without a guard the first iteration's boundary metrics (all
    equal) show in the posterior."""
    ks = [512] * 300
    llr = std_code_blocks(tc, ks, 1.5, 37)[0] if std else awgn_blocks(tc, ks, 1.5, 37)[0]
    _compare(tc, decoder, oracle, ks, 3.0 * llr, iters, std=std, guard=guard)


@pytest.mark.parametrize("std", [False, True])
@pytest.mark.parametrize("persistent", [False, True])
def test_infinite_llrs(tc, decoder, oracle, persistent, std):
    """Known bits as infinite LLRs (systematic of either sign, parities known to be 0): weights of exactly 0,
    which lose nothing.  Against 64 bits with 1e6 in their place; the known positions come back infinite."""
    rng = np.random.default_rng(38)
    ks = [40, 512, 1056, 6144, 104, 6144]
    sent = np.sign(std_code_blocks(tc, ks, 40.0, 38)[0] if std else awgn_blocks(tc, ks, 40.0, 38)[0])
    sigma2 = 1.5 / 10 ** 0.05
    llr = (2 / sigma2 * (sent + np.sqrt(sigma2) * rng.normal(size=sent.size))).astype(np.float32)
    known = np.zeros(llr.size, bool)
    lo = 0
    for k in ks:
        known[lo + 3:lo + k:17] = True
        for p in (1, 2):
            known[lo + p * (k + 4) + 5:lo + p * (k + 4) + k:31] = True
            known[lo + p * (k + 4):lo + p * (k + 4) + k] &= sent[lo + p * (k + 4):lo + p * (k + 4) + k] < 0
        lo += 3 * (k + 4)
    sched = tc.SCHEDULE_PERSISTENT if persistent else tc.SCHEDULE_PLAIN
    conv = tc.CONVENTION_3GPP if std else tc.CONVENTION_REFERENCE
    given = np.where(known, sent * np.inf, llr).astype(np.float32)
    post, _, _ = decoder.decode(ks, given, None, tc.DecodeOptions(4, False, 0, 96, sched, convention=conv))
    lo = po = 0
    for k in ks:
        x = np.where(known, sent * 1e6, llr)[lo:lo + 3 * (k + 4)]
        ref = oracle.adj_vjp(k, x, [1.0] * 8, schedule_window(k, persistent), 96, std=std)[0]
        got, at = post[po:po + k], known[lo:lo + k]
        assert np.array_equal(got[at], sent[lo:lo + k][at] * np.inf), k
        bar = np.maximum(1e-3 * np.maximum(np.abs(ref), 1.0), 2e-5 * np.abs(ref[~at]).max())
        assert (np.abs(got - ref) <= bar)[~at].all(), k
        lo += 3 * (k + 4)
        po += k
