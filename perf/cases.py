"""The work that users of the decoder have it do, as measurable cases over its public entry points.

A case names its kind and its sizes; `prepare` makes what a receiver, a link simulator or a
training job has in hand before the call, `run` is the call, `work` the bytes and operations it
cannot do without and `exact` the same function in 64-bit torch, without this library.
"""
import math

import numpy as np
import torch

import turbo_cpp_b200 as tc
from turbo_cpp_b200.autograd import DifferentiableDecoder

HARD_LIMIT = 4096 * 6144 * 8  # information bits x iterations of the largest case

# ------------------------------------------------------------------------------------------
# The code, restated: block sizes and QPP coefficients (TS 36.212 Table 5.1.3-3), CRC24B
# ------------------------------------------------------------------------------------------
SIZES = [*range(40, 513, 8), *range(528, 1025, 16), *range(1056, 2049, 32), *range(2112, 6145, 64)]
F1 = [3, 7, 19, 7, 7, 11, 5, 11, 7, 41, 103, 15, 9, 17, 9, 21, 101, 21, 57, 23, 13, 27, 11, 27, 85,
      29, 33, 15, 17, 33, 103, 19, 19, 37, 19, 21, 21, 115, 193, 21, 133, 81, 45, 23, 243, 151, 155,
      25, 51, 47, 91, 29, 29, 247, 29, 89, 91, 157, 55, 31, 17, 35, 227, 65, 19, 37, 41, 39, 185, 43,
      21, 155, 79, 139, 23, 217, 25, 17, 127, 25, 239, 17, 137, 215, 29, 15, 147, 29, 59, 65, 55, 31,
      17, 171, 67, 35, 19, 39, 19, 199, 21, 211, 21, 43, 149, 45, 49, 71, 13, 17, 25, 183, 55, 127,
      27, 29, 29, 57, 45, 31, 59, 185, 113, 31, 17, 171, 209, 253, 367, 265, 181, 39, 27, 127, 143,
      43, 29, 45, 157, 47, 13, 111, 443, 51, 51, 451, 257, 57, 313, 271, 179, 331, 363, 375, 127, 31,
      33, 43, 33, 477, 35, 233, 357, 337, 37, 71, 71, 37, 39, 127, 39, 39, 31, 113, 41, 251, 43, 21,
      43, 45, 45, 161, 89, 323, 47, 23, 47, 263]
F2 = [10, 12, 42, 16, 18, 20, 22, 24, 26, 84, 90, 32, 34, 108, 38, 120, 84, 44, 46, 48, 50, 52, 36,
      56, 58, 60, 62, 32, 198, 68, 210, 36, 74, 76, 78, 120, 82, 84, 86, 44, 90, 46, 94, 48, 98, 40,
      102, 52, 106, 72, 110, 168, 114, 58, 118, 180, 122, 62, 84, 64, 66, 68, 420, 96, 74, 76, 234,
      80, 82, 252, 86, 44, 120, 92, 94, 48, 98, 80, 102, 52, 106, 48, 110, 112, 114, 58, 118, 60,
      122, 124, 84, 64, 66, 204, 140, 72, 74, 76, 78, 240, 82, 252, 86, 88, 60, 92, 846, 48, 28, 80,
      102, 104, 954, 96, 110, 112, 114, 116, 354, 120, 610, 124, 420, 64, 66, 136, 420, 216, 444,
      456, 468, 80, 164, 504, 172, 88, 300, 92, 188, 96, 28, 240, 204, 104, 212, 192, 220, 336, 228,
      232, 236, 120, 244, 248, 168, 64, 130, 264, 134, 408, 138, 280, 142, 480, 146, 444, 120, 152,
      462, 234, 158, 80, 96, 902, 166, 336, 170, 86, 174, 176, 178, 120, 182, 184, 186, 94, 190, 480]
COEFFICIENTS = {k: (a, b) for k, a, b in zip(SIZES, F1, F2)}
CRC24B = {0: 0xC00063, 1: 0x800063}  # the library's two conventions, x^24 left out

# extrinsic scales of the size that training gives (two per iteration)
TRAINED = [0.978, 0.992, 0.985, 0.976, 0.982, 0.977, 0.981, 0.974, 0.980, 0.978, 0.984, 0.972, 0.98,
           0.976, 0.982, 0.973]


def listed():
    return [
        # one short control-sized block on the device, the smallest call: launches and latency
        dict(name="block_k40", kind="decode", n=1, k=40, iterations=8, early_stop=True,
             schedule=0, ebn0=3.0, spread=0.0),
        # one full-size block from and to host arrays, as the per-block API of the library is used
        dict(name="block_k6144_host", kind="block", k=6144, iterations=8, early_stop=False, ebn0=1.2),
        # a link simulation of short blocks, default options
        dict(name="batch_k1024", kind="decode", n=1000, k=1024, iterations=8, early_stop=False,
             schedule=0, ebn0=0.5, spread=0.0),
        # the throughput benchmark: full-size blocks over the whole waterfall, fixed iterations
        dict(name="batch_k6144", kind="decode", n=4096, k=6144, iterations=8, early_stop=False,
             schedule=1, ebn0=0.0, spread=1.2),
        # a receiver's batch under the default schedule, CRC early stop and trained scales
        dict(name="scaled_k6144", kind="decode", n=512, k=6144, iterations=8, early_stop=True,
             schedule=0, ebn0=0.8, spread=1.0, scaled=True),
        # a base station's mixed traffic: all block sizes in one call, early stop
        dict(name="mixed_20000", kind="decode", n=20000, k=0, iterations=8, early_stop=True,
             schedule=1, ebn0=0.5, spread=2.0, mix=5),
        # the TS 36.212 code, mixed odd sizes
        dict(name="std_mixed_256", kind="decode", n=256, k=0, iterations=6, early_stop=True,
             schedule=1, ebn0=1.0, spread=1.5, mix=7, convention=1),
        # one large transport block per subframe, replayed as a graph: latency of the whole chain
        dict(name="tb_one", kind="chain", n=1, least=97896, most=97896, iterations=8, schedule=0,
             graph=True, mix=1),
        # the subframes of a whole cell in one call: uneven transport blocks through the chain
        dict(name="tb_512", kind="chain", n=512, least=1000, most=97896, iterations=8, schedule=1,
             graph=False, mix=33),
        # a training step of the unrolled decoder: forward and backward
        dict(name="train_k6144", kind="train", n=1024, k=6144, iterations=6),
        # soft combining of four transmissions per code block before a retransmission's decode
        dict(name="harq_512", kind="harq", n=512, tx=4, mix=11),
        # the transmit side: turbo encoding and rate matching of mixed blocks
        dict(name="encode_4096", kind="encode", n=4096, k=0, mix=13, rate=0.5),
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    """One more case of the same ranges."""
    kind = rng.choice(["decode", "decode", "decode", "decode", "block", "chain", "train", "harq",
                       "encode"])
    mix = rng.randrange(1, 10000)
    if kind == "block":
        return dict(kind=kind, k=rng.choice(SIZES), iterations=rng.randint(1, 8),
                    early_stop=rng.random() < 0.5, ebn0=round(rng.uniform(1.0, 2.5), 2))
    if kind == "decode":
        std = rng.random() < 0.2
        k = 0 if rng.random() < 0.5 else rng.choice(SIZES)
        iterations = rng.randint(1, 8)
        most = min(256 if std else 20000, HARD_LIMIT // ((k or 6144) * iterations))
        early = rng.random() < 0.5
        c = dict(kind=kind, n=_log_int(rng, 1, most), k=k, iterations=iterations, early_stop=early,
                 schedule=rng.randrange(2), ebn0=round(rng.uniform(0.5, 2.0), 2),
                 spread=round(rng.uniform(0.0, 1.0), 2), mix=mix)
        if std:
            c["convention"] = 1
        if rng.random() < 0.25:
            c["scaled"] = True
        return c
    if kind == "chain":
        least = _log_int(rng, 1000, 20000)
        return dict(kind=kind, n=_log_int(rng, 1, 256), least=least,
                    most=_log_int(rng, least, 97896), iterations=rng.randint(4, 8),
                    schedule=rng.randrange(2), graph=rng.random() < 0.5, mix=mix)
    if kind == "train":
        k = rng.choice([k for k in SIZES if k >= 128 and k % 64 == 0])
        iterations = rng.randint(2, 6)
        return dict(kind=kind, n=_log_int(rng, 8, 1024 * 6144 * 6 // (k * iterations * 2)), k=k,
                    iterations=iterations)
    if kind == "harq":
        return dict(kind=kind, n=_log_int(rng, 8, 512), tx=rng.randint(2, 4), mix=mix)
    return dict(kind=kind, n=_log_int(rng, 16, 4096), k=0 if rng.random() < 0.7 else rng.choice(SIZES),
                mix=mix, rate=round(rng.uniform(0.34, 0.9), 2))


# ------------------------------------------------------------------------------------------
# inputs
# ------------------------------------------------------------------------------------------
_decoder = None


def decoder():
    """The program's decoder handle, created once."""
    global _decoder
    if _decoder is None:
        _decoder = tc.Decoder(0)
    return _decoder


def _block_sizes(case):
    """K per block: one size, or all sizes with larger ones more often (P ~ K), as traffic has."""
    if case.get("k"):
        return np.full(case["n"], case["k"], np.int64)
    table = np.array(SIZES)
    return np.random.default_rng(case["mix"]).choice(table, size=case["n"], p=table / table.sum())


def _ebn0(case, n, seed):
    u = np.random.default_rng([seed, 17]).uniform(0.0, 1.0, n)
    return (case["ebn0"] + case.get("spread", 0.0) * u).astype(np.float32)


def _llrs(case, ks, seed):
    """Information bits (with CRC24B where the decoder stops on it) and channel LLRs 2y/sigma^2 of
    BPSK over AWGN, [d0|d1|d2] per block back to back, on the GPU."""
    n = len(ks)
    eb = _ebn0(case, n, seed)
    conv = case.get("convention", 0)
    if conv == 0:
        return decoder().awgn_code_blocks_device(seed, ks, eb, None, bool(case.get("early_stop")))
    rng = np.random.default_rng(seed)
    words, bits = [], []
    for i, k in enumerate(ks):
        b = tc.append_crc24b(rng.integers(0, 2, int(k) - 24, dtype=np.uint8), conv)
        e = tc.turbo_encode_code_block(tc.CodeBlockDescriptor(i, int(k)), b, conv)
        words.append(np.concatenate([e.systematic, e.parity0, e.parity1]))
        bits.append(b)
    lens = 3 * (ks + 4)
    sigma2 = 1.0 / (2.0 * (ks / lens) * 10.0 ** (eb / 10.0))
    s2 = torch.from_numpy(np.repeat(sigma2, lens)).cuda()
    x = torch.from_numpy(np.concatenate(words)).cuda().double() * 2 - 1
    g = torch.Generator(device="cuda").manual_seed(seed)
    y = x + s2.sqrt() * torch.randn(x.numel(), generator=g, device="cuda", dtype=torch.float64)
    return torch.from_numpy(np.concatenate(bits)).cuda(), (2 * y / s2).float()


def _chain_sizes(case):
    """TBS and channel bits of each transport block, its code blocks (K, filler, E, rv 0), as the
    library's own segmentation gives them."""
    rng = np.random.default_rng(case["mix"])
    sizes = (rng.integers(case["least"] // 8, case["most"] // 8 + 1, case["n"]) * 8).astype(int)
    rates = rng.uniform(0.34, 0.8, case["n"])
    return sizes, rates


def _prepare_chain(case, seed):
    dec = decoder()
    sizes, rates = _chain_sizes(case)
    rng = np.random.default_rng(seed)
    tbs, blocks, payload, sigma2 = [], [], [], []
    for size, rate in zip(sizes, rates):
        with_crc = tc.append_crc24a(rng.integers(0, 2, size, dtype=np.uint8))
        seg = tc.segment_transport_block(with_crc)
        g_total = 2 * math.ceil(size / rate / 2)
        # link adaptation keeps failing transport blocks rare: an Eb/N0 above the rate's threshold
        ebn0 = 2.6 + 5.0 * (rate - 1 / 3) + rng.uniform(0.0, 1.5)
        for r, cb in enumerate(seg.code_blocks):
            e = tc.compute_e(r, g_total, seg.c, 1, 2)
            blocks.append((cb.size, seg.filler_bits if r == 0 else 0, e, 0))
            payload.append(cb)
            sigma2.append(1.0 / (2.0 * (size / g_total) * 10.0 ** (ebn0 / 10.0)))
        tbs.append((int(size), seg.c))
    blocks = np.array(blocks, np.int64)
    bits = torch.from_numpy(np.concatenate(payload)).cuda()
    d012 = dec.turbo_encode_device(blocks[:, 0], bits, blocks[:, 1])
    coded = dec.rate_match_device(blocks, d012)
    s2 = torch.from_numpy(np.repeat(np.array(sigma2), blocks[:, 2])).cuda()
    g = torch.Generator(device="cuda").manual_seed(seed)
    y = coded.double() * 2 - 1 + s2.sqrt() * torch.randn(coded.numel(), generator=g, device="cuda",
                                                         dtype=torch.float64)
    arr, e_len, _ = dec.rm_blocks(blocks)
    tba, nbits = dec.tb_descriptors(tbs)
    z = lambda m, t: torch.zeros(m, dtype=t, device="cuda")  # noqa: E731
    stream = torch.cuda.Stream() if case["graph"] else None
    return dict(e=(2 * y / s2).float(), arr=arr, n_cb=len(blocks), tba=tba, n_tb=len(tbs), e_len=e_len,
                nbits=nbits, bits=z(nbits, torch.uint8), tb_ok=z(len(tbs), torch.uint8),
                cb_ok=z(len(blocks), torch.uint8), iters=z(len(blocks), torch.int32), stream=stream,
                options=tc.DecodeOptions(case["iterations"], True, schedule=case["schedule"],
                                         graph=case["graph"]))


def _harq_transmissions(case):
    """(K, filler, E, rv, e offset, LLR offset) tuples: tx transmissions per code block."""
    ks = _block_sizes(dict(case, k=0))
    rng = np.random.default_rng([case["mix"], 1])
    out, eo, lo = [], 0, 0
    for k in ks:
        filler = int(rng.integers(0, 8)) if k > 64 else 0
        for t in range(case["tx"]):
            e = int(k / rng.uniform(0.4, 0.95))
            out.append((int(k), filler, e, (0, 2, 3, 1)[t], eo, lo))
            eo += e
        lo += 3 * (int(k) + 4)
    return out, eo, lo


def prepare(case, seed):
    kind = case["kind"]
    state = dict(case=case)
    if kind == "block":
        k = case["k"]
        _, llr = _llrs(dict(case, n=1), np.array([k]), seed)
        d = llr.cpu().numpy()
        state.update(descriptor=tc.CodeBlockDescriptor(0, k), d0=d[:k + 4].copy(),
                     d1=d[k + 4:2 * k + 8].copy(), d2=d[2 * k + 8:].copy())
    elif kind == "decode":
        ks = _block_sizes(case)
        bits, llr = _llrs(case, ks, seed)
        cbs, llr_len, post_len = tc.Decoder.layout(ks)
        n = len(ks)
        scales = TRAINED[:2 * case["iterations"]] if case.get("scaled") else None
        state.update(cbs=cbs, n=n, llr=llr, llr_len=llr_len, post_len=post_len,
                     post=torch.zeros(post_len, dtype=torch.float32, device="cuda"),
                     crc=torch.zeros(n, dtype=torch.uint8, device="cuda"),
                     iters=torch.zeros(n, dtype=torch.int32, device="cuda"),
                     options=tc.DecodeOptions(case["iterations"], case["early_stop"],
                                              schedule=case["schedule"], scales=scales,
                                              convention=case.get("convention", 0)))
    elif kind == "chain":
        state.update(_prepare_chain(case, seed))
    elif kind == "train":
        ks = [case["k"]] * case["n"]
        bits, llr = decoder().awgn_code_blocks_device(seed, ks, 0.6)
        state.update(dd=DifferentiableDecoder(ks, decoder=decoder()), bits=bits.float(),
                     llr=llr.requires_grad_(True),
                     scales=torch.tensor(TRAINED[:2 * case["iterations"]], device="cuda",
                                         requires_grad=True))
    elif kind == "harq":
        tx, e_len, llr_len = _harq_transmissions(case)
        g = torch.Generator(device="cuda").manual_seed(seed)
        sign = torch.randint(0, 2, (e_len,), generator=g, device="cuda") * 2.0 - 1.0
        e = 4.0 * sign + 2.8 * torch.randn(e_len, generator=g, device="cuda")
        state.update(tx=tx, e=e, e_len=e_len, llr_len=llr_len,
                     out=torch.zeros(llr_len, dtype=torch.float32, device="cuda"))
    else:
        ks = _block_sizes(case)
        g = torch.Generator(device="cuda").manual_seed(seed)
        bits = torch.randint(0, 2, (int(ks.sum()),), generator=g, device="cuda", dtype=torch.uint8)
        blocks = np.stack([ks, np.zeros_like(ks), (ks / case["rate"]).astype(np.int64),
                           np.arange(len(ks)) % 4], 1)
        state.update(ks=ks, bits=bits, blocks=blocks)
    return state


def run(state):
    kind, dec = state["case"]["kind"], decoder()
    s = state
    if kind == "block":
        post, ok, it = tc.turbo_decode_code_block_gpu(s["descriptor"], s["d0"], s["d1"], s["d2"],
                                                      s["case"]["iterations"],
                                                      s["case"]["early_stop"])
        return dict(posterior=post, ok=ok, iterations=it)
    if kind == "decode":
        dec.decode_device(s["cbs"], s["n"], s["llr"].data_ptr(), s["llr_len"], s["post"].data_ptr(),
                          s["post_len"], s["crc"].data_ptr(), s["iters"].data_ptr(), s["options"])
        return dict(posterior=s["post"], ok=s["crc"], iterations=s["iters"])
    if kind == "chain":
        stream = s["stream"].cuda_stream if s["stream"] is not None else 0
        dec.decode_tbs_device(s["tba"], s["n_tb"], s["arr"], s["n_cb"], s["e_len"], s["e"].data_ptr(),
                              s["nbits"], s["bits"].data_ptr(), s["tb_ok"].data_ptr(),
                              s["cb_ok"].data_ptr(), s["iters"].data_ptr(), s["options"], stream)
        return dict(bits=s["bits"], tb_ok=s["tb_ok"], cb_ok=s["cb_ok"], iterations=s["iters"])
    if kind == "train":
        post = s["dd"](s["llr"], s["scales"])
        loss = torch.nn.functional.binary_cross_entropy_with_logits(post, s["bits"], reduction="sum")
        g_llr, g_scales = torch.autograd.grad(loss, [s["llr"], s["scales"]])
        return dict(posterior=post.detach(), grad_llr=g_llr, grad_scales=g_scales)
    if kind == "harq":
        dec.derate_combine_device(s["tx"], s["e"].data_ptr(), s["e_len"], s["out"].data_ptr(),
                                  s["llr_len"])
        return s["out"]
    d012 = dec.turbo_encode_device(s["ks"], s["bits"])
    return dict(encoded=d012, rate_matched=dec.rate_match_device(s["blocks"], d012))


def work(case):
    """Inputs read once, outputs written once; per trellis step of a SISO two 8-state recursions of
    three operations a state and an extrinsic of 32, a decode with early stop taken as half its
    iterations (the gradient step as three times its forward pass)."""
    kind = case["kind"]
    if kind == "harq":
        _, e_len, llr_len = _harq_transmissions(case)
        return dict(bytes=4 * e_len + 4 * llr_len, flops=e_len)
    if kind == "chain":
        sizes, rates = _chain_sizes(case)
        return dict(bytes=float((4 * sizes / rates + sizes).sum()),
                    flops=float(sizes.sum()) * 80 * case["iterations"])
    ks = np.array([case["k"]]) if kind == "block" else _block_sizes(case)
    bits = int(ks.sum())
    if kind == "encode":
        return dict(bytes=bits * (1 + 3 + 1 / case["rate"]), flops=8 * bits)
    llrs = 3 * (bits + 4 * len(ks))
    steps = 2.0 * bits * case["iterations"]
    if kind == "train":
        return dict(bytes=4 * (2 * llrs + 2 * bits), flops=3 * 80 * steps)
    return dict(bytes=4 * (llrs + bits) + 5 * len(ks),
                flops=80 * steps * (0.5 if case["early_stop"] else 1.0))


# ------------------------------------------------------------------------------------------
# the same functions in 64 bits
# ------------------------------------------------------------------------------------------
def _qpp(k):
    f1, f2 = COEFFICIENTS[int(k)]
    i = np.arange(int(k), dtype=np.int64)
    return (f1 * i + f2 * i * i) % int(k)


def _branch_signs(std, dev):
    """Signs of the systematic and the parity term of the branch from state 2j + x to state
    4 n2 + j, as [n2, j, x]."""
    n2, j, x = np.meshgrid(np.arange(2), np.arange(4), np.arange(2), indexing="ij")
    n1, n0 = j >> 1, j & 1
    u = n2 ^ n0 ^ x if std else n2 ^ n1 ^ n0
    p = n2 ^ n1 ^ x
    return [torch.from_numpy(2.0 * v - 1.0).to(dev) for v in (u, p)]


def _tail(d0, d1, d2, lower, std):
    """beta at the block end from the 12 tail LLRs (each of d0, d1, d2: [B, 4])."""
    a, b, c = d0.unbind(1), d1.unbind(1), d2.unbind(1)
    zero = torch.zeros_like(a[0])
    if std:
        o = 2 if lower else 0
        ts, tp = (a[o], c[o], b[o + 1]), (b[o], a[o + 1], c[o + 1])
    elif lower:
        ts, tp = (b[3], c[0], c[2]), (c[1], a[3], c[3])
    else:
        ts, tp = (a[0], a[2], zero), (b[0], a[1], b[2])
    beta = []
    for state in range(8):
        s, m = state, 0.0
        for i in range(3):
            s0, s1, s2 = s & 1, (s >> 1) & 1, s >> 2
            u = s0 ^ s1 if std else s1 ^ s2
            m = m + (ts[i] if u else -ts[i]) + (tp[i] if s0 ^ s2 else -tp[i])
            s = s >> 1
        beta.append(0.5 * m)
    return torch.stack(beta, 1)


class _Blocks:
    """Code blocks padded to the longest, [B, Kmax] each, in 64 bits."""

    def __init__(self, ks, llr):
        ks = torch.as_tensor(np.asarray(ks), device=llr.device)
        n, kmax = len(ks), int(ks.max())
        start = torch.cumsum(3 * (ks + 4), 0) - 3 * (ks + 4)
        at = torch.arange(kmax, device=llr.device)[None]
        self.mask = at < ks[:, None]
        x = llr.detach().double()

        def stream(j):
            return torch.where(self.mask, x[(start[:, None] + j * (ks + 4)[:, None] + at).clamp(max=x.numel() - 1)], 0.0)

        def tail(j):
            return x[start[:, None] + j * (ks + 4)[:, None] + ks[:, None] + torch.arange(4, device=llr.device)]

        self.sys, self.par0, self.par1 = stream(0), stream(1), stream(2)
        self.tails = tail(0), tail(1), tail(2)
        perm = torch.arange(kmax, device=llr.device).repeat(n, 1)
        for k in torch.unique(ks).tolist():
            perm[ks == k, :k] = torch.from_numpy(_qpp(k)).to(llr.device)
        self.ks, self.perm, self.n, self.kmax = ks, perm, n, kmax


def _siso64(sys, par, apr, tail, ks, std):
    """Extrinsic LLRs of one SISO over the full trellis, [B, K]."""
    n, kmax = sys.shape
    su, sp = _branch_signs(std, sys.device)
    half = 0.5 * (sys + apr).t().contiguous()
    halfp = 0.5 * par.t().contiguous()
    al = sys.new_full((kmax + 1, n, 8), -math.inf)
    al[0, :, 0] = 0.0
    chunk = 128
    for t0 in range(0, kmax, chunk):
        t1 = min(t0 + chunk, kmax)
        g = half[t0:t1, :, None, None, None] * su + halfp[t0:t1, :, None, None, None] * sp
        for t in range(t0, t1):
            c = al[t].view(n, 1, 4, 2) + g[t - t0]
            torch.logaddexp(c[..., 0], c[..., 1], out=al[t + 1].view(n, 2, 4))
    ends = {k: (ks == k).nonzero()[:, 0] for k in torch.unique(ks).tolist()}
    ext = torch.empty_like(sys)
    be = sys.new_zeros((chunk + 1, n, 8))
    for t1 in range(kmax, 0, -chunk):
        t0 = max(t1 - chunk, 0)
        g = half[t0:t1, :, None, None, None] * su + halfp[t0:t1, :, None, None, None] * sp
        be[t1 - t0] = be[0].clone() if t1 < kmax else 0.0
        for t in range(t1 - 1, t0 - 1, -1):
            if t + 1 in ends:
                be[t + 1 - t0, ends[t + 1]] = tail[ends[t + 1]]
            nxt = be[t + 1 - t0].view(n, 2, 4).unsqueeze(-1)
            c = nxt + g[t - t0]
            torch.logaddexp(c[:, 0], c[:, 1], out=be[t - t0].view(n, 4, 2))
        m = (al[t0:t1].view(-1, n, 1, 4, 2) + be[1:t1 - t0 + 1].view(-1, n, 2, 4, 1)
             + halfp[t0:t1, :, None, None, None] * sp).reshape(t1 - t0, n, 16)
        one = (su > 0).reshape(16)
        ext[:, t0:t1] = (torch.logsumexp(m[..., one], -1) - torch.logsumexp(m[..., ~one], -1)).t()
    return ext


def _crc_ok(hard, ks, mask):
    """CRC24B over the K hard decisions of each block."""
    r, rows = 1, []
    for _ in range(int(ks.max())):
        rows.append([(r >> b) & 1 for b in range(24)])
        r <<= 1
        if r >> 24:
            r ^= (1 << 24) | mask
    table = torch.tensor(rows, dtype=torch.float64, device=hard.device)
    ok = torch.zeros(len(ks), dtype=torch.bool, device=hard.device)
    for k in torch.unique(ks).tolist():
        at = ks == k
        ok[at] = ((hard[at, :k].double() @ table[:k].flip(0)) % 2 == 0).all(1)
    return ok


def _exact_decode(case, ks, llr):
    """Full-trellis Log-MAP iterations; a block keeps the posterior of the iteration it stops at."""
    b = _Blocks(ks, llr)
    std = case.get("convention", 0) == 1
    scales = TRAINED if case.get("scaled") else [1.0] * 16
    tails = [_tail(*b.tails, lower, std) for lower in (False, True)]
    sys_i = torch.gather(b.sys, 1, b.perm)
    e2 = torch.zeros_like(b.sys)
    post, running = torch.zeros_like(b.sys), torch.ones(b.n, dtype=torch.bool, device=llr.device)
    for it in range(case["iterations"]):
        e1 = scales[2 * it] * _siso64(b.sys, b.par0, e2, tails[0], b.ks, std)
        e1i = torch.gather(e1, 1, b.perm)
        e2i = scales[2 * it + 1] * _siso64(sys_i, b.par1, e1i, tails[1], b.ks, std)
        e2 = torch.zeros_like(e2i).scatter_(1, b.perm, e2i)
        post[running] = (b.sys + e1 + e2)[running]
        if case["early_stop"]:
            running &= ~_crc_ok(post >= 0, b.ks, CRC24B[int(std)])
            if not bool(running.any()):
                break
    return post[b.mask]


def _window_siso(apr, sys, par, tail, seed_a, seed_b, w, g):
    """One SISO of the differentiable schedule: windows of w steps with warm-ups of g steps from
    fixed seeds.  Returns the extrinsic and the seeds for the next iteration."""
    n, k = sys.shape
    nw = k // w
    su, sp = _branch_signs(False, sys.device)
    pad = lambda v: torch.nn.functional.pad(v, (g, w + g))  # noqa: E731
    at = torch.arange(nw, device=sys.device)[:, None] * w + torch.arange(w + 2 * g, device=sys.device)
    half, halfp = 0.5 * pad(sys + apr)[:, at], 0.5 * pad(par)[:, at]  # [n, nw, w + 2g]
    step = lambda s: half[:, :, s, None, None, None] * su + halfp[:, :, s, None, None, None] * sp  # noqa: E731
    start = torch.full((8,), -1e30, dtype=sys.dtype, device=sys.device)
    start[0] = 0.0
    a, als = seed_a, []
    for s in range(w + g):
        if (g - s) % w == 0 and 0 <= (g - s) // w < nw:  # the block start
            v = (g - s) // w
            a = torch.cat([a[:, :v], start.expand(n, 1, 8), a[:, v + 1:]], 1)
        als.append(a)
        c = a.view(n, nw, 1, 4, 2) + step(s)
        a = torch.logaddexp(c[..., 0], c[..., 1]).reshape(n, nw, 8)
    be, bes = seed_b, {}
    for s in range(w + g - 1, -1, -1):
        if (k - 1 - s) % w == 0 and 0 <= (k - 1 - s) // w < nw:  # the block end
            v = (k - 1 - s) // w
            be = torch.cat([be[:, :v], tail[:, None], be[:, v + 1:]], 1)
        bes[s] = be
        c = be.view(n, nw, 2, 4, 1) + step(s + g)
        be = torch.logaddexp(c[:, :, 0], c[:, :, 1]).reshape(n, nw, 8)
    al_own = torch.stack(als[g:], 2).view(n, nw, w, 1, 4, 2)
    be_own = torch.stack([bes[s] for s in range(w)], 2).view(n, nw, w, 2, 4, 1)
    m = (al_own + be_own + halfp[:, :, g:g + w, None, None, None] * sp).reshape(n, nw, w, 16)
    one = (su > 0).reshape(16)
    ext = torch.logsumexp(m[..., one], -1) - torch.logsumexp(m[..., ~one], -1)
    zero = seed_a.new_zeros(n, 1, 8)
    next_a = torch.cat([zero, als[w][:, :-1]], 1).detach()  # alpha at the next window's warm-up start
    next_b = torch.cat([bes[g - 1][:, 1:], zero], 1).detach()
    return ext.reshape(n, k), next_a, next_b


def _exact_train(case, seed):
    state = prepare(case, seed)
    from torch.utils.checkpoint import checkpoint

    k, n, w, g = case["k"], case["n"], 64, 32
    scales = state["scales"].detach().double().requires_grad_(True)
    perm = torch.from_numpy(_qpp(k)).cuda()
    inv = torch.argsort(perm)
    posts, grads, per = [], [], max(1, 128 * 6144 // k)
    g_scales = torch.zeros_like(scales)
    for i in range(0, n, per):
        m = min(per, n - i)
        x = state["llr"].detach().view(n, 3 * (k + 4))[i:i + m].double().requires_grad_(True)
        d0, d1, d2 = x.split(k + 4, 1)
        tails = [_tail(d0[:, k:], d1[:, k:], d2[:, k:], lower, False) for lower in (False, True)]
        sys, e2 = d0[:, :k], torch.zeros_like(d0[:, :k])
        zero = x.new_zeros(m, k // w, 8)
        seeds = [(zero, zero), (zero, zero)]
        for it in range(case["iterations"]):
            e, *seeds[0] = checkpoint(_window_siso, e2, sys, d1[:, :k], tails[0], *seeds[0], w, g,
                                      use_reentrant=False)
            e1 = scales[2 * it] * e
            e, *seeds[1] = checkpoint(_window_siso, e1[:, perm], sys[:, perm], d2[:, :k], tails[1],
                                      *seeds[1], w, g, use_reentrant=False)
            e2 = (scales[2 * it + 1] * e)[:, inv]
        post = sys + e1 + e2
        bits = state["bits"].view(n, k)[i:i + m].double()
        loss = torch.nn.functional.binary_cross_entropy_with_logits(post, bits, reduction="sum")
        gx, gs = torch.autograd.grad(loss, [x, scales])
        posts.append(post.detach())
        grads.append(gx)
        g_scales += gs
    return dict(posterior=torch.cat(posts).reshape(-1), grad_llr=torch.cat(grads).reshape(-1),
                grad_scales=g_scales)


def _circular_sources(k, filler):
    """The circular buffer: index into [d0|d1|d2] of each position that is not <NULL>, and the
    buffer's length, rows and validity."""
    d = k + 4
    rows = -(-d // 32)
    kpi = 32 * rows
    column = np.array([int(f"{c:05b}"[::-1], 2) for c in range(32)])
    row = np.arange(rows)
    first = (32 * row[None, :] + column[:, None]).reshape(-1) - (kpi - d)  # column by column
    last = (column[:, None] + 32 * row[None, :] + 1).reshape(-1) % kpi - (kpi - d)
    v0 = np.where(first < filler, -1, first)
    v1 = np.where(first < filler, -1, d + first)
    v2 = np.where(last < 0, -1, 2 * d + last)
    v0[first < 0] = -1
    return np.concatenate([v0, np.stack([v1, v2], 1).reshape(-1)]), rows


def _exact_harq(case, seed):
    state = prepare(case, seed)
    e = state["e"].cpu().numpy().astype(np.float64)
    out = np.zeros(state["llr_len"])
    for k, filler, n, rv, eo, lo in state["tx"]:
        src, rows = _circular_sources(k, filler)
        k0 = rows * (2 * -(-len(src) // (8 * rows)) * rv + 2) % len(src)
        src = np.roll(src, -k0)
        src = src[src >= 0]
        np.add.at(out, lo + src[np.arange(n) % len(src)], e[eo:eo + n])
    return torch.from_numpy(out)


def exact(case, seed):
    kind = case["kind"]
    if kind == "block":
        _, llr = _llrs(dict(case, n=1), np.array([case["k"]]), seed)
        return dict(posterior=_exact_decode(case, [case["k"]], llr), ok=None, iterations=None)
    if kind == "decode":
        ks = _block_sizes(case)
        _, llr = _llrs(case, ks, seed)
        return dict(posterior=_exact_decode(case, ks, llr), ok=None, iterations=None)
    if kind == "train":
        return _exact_train(case, seed)
    if kind == "harq":
        return _exact_harq(case, seed)
    return None  # whole numbers only
