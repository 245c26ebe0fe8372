"""The device encoder (32 steps per thread) and rate matcher (by rank, 4 bits per store) against the
host codec, bit for bit: block sizes around whole words, warps of words and the largest; fillers
around words; streams at every byte alignment; outputs from one bit to several times the buffer."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

KS = [40, 48, 64, 992, 1008, 1024, 1056, 6080, 6144]


def _encoded(tc, ks, fillers, seed):
    bits = [tc.random_bits(seed + i, k) for i, k in enumerate(ks)]
    host = []
    for k, f, b in zip(ks, fillers, bits):
        b[:f] = 0
        e = tc.turbo_encode_code_block(tc.CodeBlockDescriptor(k_r=k, filler_count=f), b)
        host.append(np.concatenate([e.systematic, e.parity0, e.parity1]))
    return np.concatenate(bits), np.concatenate(host)


@pytest.mark.parametrize("shift", [0, 1, 2, 3])
@pytest.mark.parametrize("filler", [0, 1, 31, 32, 33])
def test_encoder(tc, decoder, filler, shift):
    import torch

    bits, host = _encoded(tc, KS, [filler] * len(KS), 40 + filler)
    ks = np.array(KS, np.int32)
    fl = np.full(ks.size, filler, np.int32)
    x = torch.zeros(bits.size + 4, dtype=torch.uint8, device="cuda")
    x[shift:shift + bits.size] = torch.from_numpy(bits).cuda()
    d = decoder.turbo_encode_device(ks, x[shift:shift + bits.size], fl)
    assert np.array_equal(d.cpu().numpy(), host)


@pytest.mark.parametrize("rv", [0, 1, 2, 3])
def test_rate_matcher(tc, decoder, rv):
    import torch

    blocks = []
    for i, k in enumerate(KS):
        for e in (1, 2, 3, 4, 5, 7, k, 3 * (k + 4), 7 * k + 3):
            blocks.append((k, (0, 8, k - 1)[(i + e) % 3], e, rv))
    _, host = _encoded(tc, [b[0] for b in blocks], [b[1] for b in blocks], 90)
    out = decoder.rate_match_device(blocks, torch.from_numpy(host).cuda()).cpu().numpy()
    lo = pos = 0
    for k, f, e, r in blocks:
        assert np.array_equal(out[lo:lo + e], tc.rate_match(k, f, host[pos:pos + 3 * (k + 4)], e, r)), (k, f, e)
        lo += e
        pos += 3 * (k + 4)


@pytest.mark.parametrize("form", ["tuples", "array", "floats"])
def test_combining_takes_any_number_type(tc, decoder, form):
    """Soft combining's descriptors as tuples of int, rows of an integer array, or floats."""
    import torch

    rng = np.random.default_rng(5)
    tx, eo, lo = [], 0, 0
    for k in (40, 1056):
        for rv in range(3):
            tx.append((k, 8, 2 * k, rv, eo, lo))
            eo += 2 * k
        lo += 3 * (k + 4)
    e = torch.from_numpy(rng.normal(size=eo).astype(np.float32)).cuda()
    ref = np.zeros(lo)
    for k, f, n, rv, at, out in tx:
        one = torch.zeros(lo, device="cuda")
        decoder.derate_combine_device([(k, f, n, rv, at, 0)], e.data_ptr(), eo, one.data_ptr(), 3 * (k + 4))
        torch.cuda.synchronize()
        ref[out:out + 3 * (k + 4)] += one.cpu().numpy()[:3 * (k + 4)]
    given = {"tuples": tx, "array": np.array(tx), "floats": [tuple(float(v) for v in t) for t in tx]}[form]
    got = torch.zeros(lo, device="cuda")
    decoder.derate_combine_device(given, e.data_ptr(), eo, got.data_ptr(), lo)
    torch.cuda.synchronize()
    # three sums of float32 values of size 1 to 5, in another order: 3 roundings of 2^-24 x 15
    assert np.abs(got.cpu().numpy() - ref).max() <= 3e-6
