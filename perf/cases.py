"""Performance cases of the decoder: what its callers run, through the public
entry points of ``dvc_b200.native``, from a single bitplane to many streams.

    listed()            the named cases
    draw(rng)           one more case of the same ranges
    prepare(case, seed) the inputs of a case (bitplanes or streams) and its handle
    run(state)          one pass: the call a program makes, with its outputs
    work(case)          bytes and operations a pass cannot do without
    exact(case, seed)   float outputs in 64-bit arithmetic

A case is a dict whose "call" names the entry point:

* "bitplane": ``Context.LdpcaDecoder``, the drop-in for the reference's own
  per-bitplane call (one codeword, the caller's rate bound).
* "codewords": ``Context.ldpca_decode``, equal-length codewords in one call.
* "mixed": ``Context.ldpca_decode_batch``, codewords of both lengths, each from
  its own start level.
* "encode": ``Context.ldpca_encode``, the encoder's side of the same codes.
* "frames": ``Context.decode_wz_frames``, the plain decode of one or more
  independent frames with host buffers in and out.
* "session": ``Context.session``, whole sequences resident on the device,
  decoded by every run and read back.
* "serve": ``Context.server``, single-frame requests of many streams.

Codewords carry likelihood ratios that vary from bit to bit as a Laplacian
correlation-noise model gives them, clipped where the decoder clips them.
Frames come from the package's synthetic sequences and its encoder.  "tools"
switches SkipBlock, IntraMode and DeblockingFilter on together, as the CIF
benchmark configuration has them; every other stream with tools is then a
still-camera one, whose frames have skip blocks.
"""
import functools
import os
import time

# one hardware queue per CUDA stream, as the package's own programs set it
os.environ.setdefault("CUDA_DEVICE_MAX_CONNECTIONS", "32")

import numpy as np  # noqa: E402

from dvc_b200 import bitstream, decoder, encoder, intra, ldpca_bench, native, synth  # noqa: E402

SIZES = {"qcif": (176, 144), "cif": (352, 288)}
LENGTHS = {"qcif": 1584, "cif": 6336}
INTRA_QP = 30


def listed():
    return [
        # one bitplane through the drop-in call: the smallest request, latency counts
        dict(name="bitplane_qcif", call="bitplane", size="qcif", noise=0.05),
        dict(name="bitplane_cif", call="bitplane", size="cif", noise=0.11),
        # the bitplanes of a few QCIF frames, fewer codewords than the device has SMs
        dict(name="codewords_qcif", call="codewords", size="qcif", count=33, noise=0.08),
        # more CIF codewords than SMs, not a multiple of them
        dict(name="codewords_cif", call="codewords", size="cif", count=203, noise=0.12),
        # thousands of codewords of both lengths from seeded start levels
        dict(name="codewords_mixed", call="mixed", count=1501, noise=0.12),
        # the encoder's syndromes for the bitplanes of ten CIF frames
        dict(name="encode_cif", call="encode", size="cif", count=300),
        # one frame of each size alone: what a plain decoder waits for
        dict(name="frame_qcif", call="frames", size="qcif", frames=1, q=3, tools=False),
        dict(name="frame_cif", call="frames", size="cif", frames=1, q=4, tools=False),
        # a level of independent frames at the highest rate, every block Wyner-Ziv coded
        dict(name="frames_cif_high", call="frames", size="cif", frames=11, q=8, tools=False),
        # sequences on the device with skip and intra blocks and the deblocking
        # filter, GOP 4 in two levels, low to high rates
        dict(name="session_cif", call="session", size="cif", gop=4, frames=17, streams=4, q=2, tools=True),
        # GOP 8 sequences of the small size in three levels
        dict(name="session_qcif", call="session", size="qcif", gop=8, frames=17, streams=3, q=4, tools=False),
        # requests of mixed streams: QCIF without tools, CIF with them
        dict(name="serve_mixed", call="serve", qcif=40, cif=14, q=1),
    ]


def _log_int(rng, lo, hi):
    """An integer spread evenly over the logarithm of [lo, hi]."""
    return min(hi, max(lo, int(round(lo * (hi / lo) ** rng.random()))))


def draw(rng):
    call = rng.choice(["bitplane", "codewords", "codewords", "mixed", "encode", "frames", "frames", "session",
                       "session", "serve"])
    size = rng.choice(["qcif", "cif"])
    noise = round(rng.uniform(0.02, 0.15), 4)
    if call == "bitplane":
        return dict(call=call, size=size, noise=noise)
    if call == "codewords":
        return dict(call=call, size=size, count=_log_int(rng, 1, 203 if size == "cif" else 600), noise=noise)
    if call == "mixed":
        return dict(call=call, count=_log_int(rng, 2, 1501), noise=noise)
    if call == "encode":
        return dict(call=call, size=size, count=_log_int(rng, 1, 300))
    if call == "frames":
        return dict(call=call, size=size, frames=_log_int(rng, 1, 11), q=rng.randint(1, 8), tools=rng.random() < 0.5)
    if call == "session":
        tools = rng.random() < 0.5
        return dict(call=call, size=size, gop=rng.choice([2, 4, 8]), frames=rng.choice([9, 13, 17]),
                    streams=rng.randint(1, 3 if tools else 2), q=rng.randint(1, 8), tools=tools)
    return dict(call=call, qcif=rng.randint(3, 40), cif=rng.randint(1, 14), q=rng.randint(1, 4))


# ------------------------------------------------------------------- inputs

@functools.lru_cache(maxsize=None)
def _context():
    """The program's decoder context, one for its lifetime."""
    return native.Context(0)


def _bits(n, count, noise, rng):
    """Source bits and the likelihood ratios p0/p1 a decoder holds for them:
    bit k is wrong in the side information with probability p_k, exponentially
    distributed around the codeword's noise level."""
    x = rng.integers(0, 2, (count, n), dtype=np.uint8)
    level = noise * rng.uniform(0.3, 1.3, (count, 1))
    p = np.clip(level * rng.standard_exponential((count, n), dtype=np.float32), 1e-4, 0.49)
    y = x ^ (rng.random((count, n), dtype=np.float32) < p)
    lr = np.where(y == 0, (1.0 - p) / p, p / (1.0 - p))
    return x, np.clip(lr, 1e-4 / 0.9999, 0.9999 / 1e-4).astype(np.float32)


def _entropy(lr):
    """Conditional entropy per bit of each row of likelihood ratios, in 64 bits."""
    p = lr.astype(np.float64) / (1.0 + lr.astype(np.float64))
    return -(p * np.log2(p) + (1.0 - p) * np.log2(1.0 - p)).mean(axis=1)


def _codewords(size, count, noise, rng):
    x, lr = _bits(LENGTHS[size], count, noise, rng)
    acc, crc = _context().ldpca_encode(x)
    return lr, acc, crc


def _stream(size, frames, gop, q, tools, seed, still=False):
    """The WZ frames of one encoded sequence as session items, in level order."""
    ori, key = synth.make_sequence(size + "_still" if still else size, frames, seed)
    if tools:
        wz, ib = encoder.encode_sequence_intra(ori, gop, q, INTRA_QP, 1, 1, 1)
    else:
        wz, ib = encoder.encode_sequence(ori, gop, q), b""
    st = bitstream.parse_wz(wz)
    start = np.array(key, np.uint8, copy=True)
    if ib:
        for m, (px, _) in intra.decode_all(st, ib, key).items():
            start[m] = px
    items, where = [], {}
    for level in decoder.decode_levels(st):
        for (m, past, future) in level:
            it = decoder.frame_item(st, st.frames[m], start)
            for name, ref in (("past", past), ("future", future)):
                if ref in st.frames:
                    it[name + "_from"], it[name] = where[ref], None
            where[m] = len(items)
            items.append(it)
    return items


def _qs(case, k):
    """The quantiser of the k-th stream: from the case's up, wrapping at 8."""
    return 1 + (case["q"] - 1 + 2 * k) % 8


def prepare(case, seed):
    rng = np.random.default_rng(seed)
    ctx = _context()
    call = case["call"]
    if call == "bitplane":
        lr, acc, crc = _codewords(case["size"], 1, case["noise"], rng)
        return dict(call=call, ctx=ctx, lr=lr[0], acc=np.unpackbits(acc[0]), crc=int(crc[0]),
                    bound=float(_entropy(lr)[0]))
    if call == "codewords":
        lr, acc, crc = _codewords(case["size"], case["count"], case["noise"], rng)
        return dict(call=call, ctx=ctx, lr=lr, acc=acc, crc=crc)
    if call == "mixed":
        count = case["count"]
        n = np.where(np.arange(count) % 2 == 0, LENGTHS["qcif"], LENGTHS["cif"]).astype(np.int32)
        lr, acc = [None] * count, [None] * count
        crc, start = np.zeros(count, np.uint8), np.zeros(count, np.int32)
        for size, first in (("qcif", 0), ("cif", 1)):
            mine = range(first, count, 2)
            if not len(mine):
                continue
            l, a, c = _codewords(size, len(mine), case["noise"], rng)
            rates = ldpca_bench.code_rates(LENGTHS[size]).astype(np.float64)
            # a request level near the entropy, as the batched benchmark seeds it
            s = np.searchsorted(rates, _entropy(l)) + rng.integers(-1, 4, len(mine))
            crc[first::2], start[first::2] = c, np.clip(s, 0, len(rates) - 2)
            for i, k in enumerate(mine):
                lr[k], acc[k] = l[i], a[i]
        return dict(call=call, ctx=ctx, n=n, lr=np.concatenate(lr), acc=np.concatenate(acc), crc=crc, start=start)
    if call == "encode":
        return dict(call=call, ctx=ctx, bits=rng.integers(0, 2, (case["count"], LENGTHS[case["size"]]), dtype=np.uint8))
    if call == "frames":
        items = _stream(case["size"], 2 * case["frames"] + 1, 2, case["q"], case["tools"], seed)
        return dict(call=call, ctx=ctx, items=items)
    if call == "session":
        items = []
        for k in range(case["streams"]):
            own = _stream(case["size"], case["frames"], case["gop"], _qs(case, k), case["tools"], seed + 101 * k,
                          still=case["tools"] and k % 2 == 1)
            for it in own:
                for name in ("past_from", "future_from"):
                    if name in it:
                        it[name] += len(items)
            items += own
        return dict(call=call, session=ctx.session(items, max_batch=16, streams=8), count=len(items))
    items = []
    for size, tools in (("qcif", False), ("cif", True)):
        left, k = case[size], 0
        while left > 0:  # streams of up to four independent frames
            n = min(4, left)
            items += _stream(size, 2 * n + 1, 2, _qs(case, k), tools, seed + 101 * k + (50 if tools else 0),
                             still=tools and k % 2 == 1)
            left, k = left - n, k + 1
    order = rng.permutation(len(items))
    return dict(call=call, server=ctx.server(mem_budget_bytes=16 << 30, streams=16, max_cohort=16),
                items=[items[i] for i in order])


# --------------------------------------------------------------------- runs

def _frame_outputs(outs):
    """Decoded pixels of all frames in order, rates and the ladder result of
    every bitplane.  The fourth number of a bitplane's result counts the BP
    iterations run, which is no output: it depends on the speculation and on
    the device's timing."""
    return dict(recon=np.concatenate([o["recon"].reshape(-1) for o in outs]), wz_bits=np.array([o["wz_bits"] for o in outs]),
                planes=np.concatenate([o["planes"] for o in outs])[:, :3])


def run(state):
    call = state["call"]
    if call == "bitplane":
        bits, rate, llr = state["ctx"].LdpcaDecoder(state["lr"], state["acc"], state["crc"], state["bound"])
        return dict(bits=bits, rate=rate, llr=llr)
    if call == "codewords":
        bits, results, entropy = state["ctx"].ldpca_decode(state["lr"], state["acc"], state["crc"])
        return dict(bits=bits, results=results, entropy=entropy)
    if call == "mixed":
        bits, results, entropy, _, _ = state["ctx"].ldpca_decode_batch(state["n"], state["lr"], state["acc"],
                                                                       state["crc"], state["start"])
        return dict(bits=bits, results=results, entropy=entropy)
    if call == "encode":
        acc, crc = state["ctx"].ldpca_encode(state["bits"])
        return dict(acc=acc, crc=crc)
    if call == "frames":
        outs = state["ctx"].decode_wz_frames(state["items"])
        return dict(_frame_outputs(outs), entropy=np.concatenate([o["entropy"] for o in outs]),
                    deblock_flag=np.stack([o["deblock_flag"] for o in outs]))
    if call == "session":
        state["session"].run()
        frames = [state["session"].frame(i) for i in range(state["count"])]
        return _frame_outputs([dict(recon=r, wz_bits=b, planes=p) for r, b, p in frames])
    server = state["server"]
    tickets = [server.submit(it) for it in state["items"]]
    outs = {}
    while len(outs) < len(tickets):
        if server.poll():
            for t in server.finished():
                outs[t] = server.result(t)
        else:
            time.sleep(0.0002)
    return _frame_outputs([outs[t] for t in tickets])


# ------------------------------------------------------- what a pass needs

def _codeword_work(n):
    """One codeword decoded by one ladder code in the shortest run, a single BP
    iteration: per edge a message each way (about 8 operations with its
    magnitude function), its ratios, syndrome and bits moved once."""
    e = 3 * n
    return dict(bytes=n * 4 + n // 8 + n, flops=2 * 8 * e)


def _frame_work(size, q):
    """One frame: both references, the bitplanes and the starting content in,
    the decoded frame out; per bitplane a codeword; per band the search of
    65x65 positions in two references at 16 pixels a block (two operations a
    pixel)."""
    w, h = SIZES[size]
    n = w * h // 16
    planes = int(sum(bitstream.QBITS[q]))
    bands = int(sum(1 for b in bitstream.QBITS[q] if b > 0))
    return dict(bytes=4 * w * h + planes * (n // 8 + 1),
                flops=planes * _codeword_work(n)["flops"] + bands * n * 2 * 65 * 65 * 16 * 2)


def _sum(works):
    works = list(works)
    return dict(bytes=sum(w["bytes"] for w in works), flops=sum(w["flops"] for w in works))


def _wz_frames(frames, gop):
    return sum(len(bitstream.gop_order(i, min(i + gop, frames - 1))) for i in range(0, frames, gop))


def work(case):
    call = case["call"]
    if call == "bitplane":
        return _codeword_work(LENGTHS[case["size"]])
    if call == "codewords":
        return _sum([_codeword_work(LENGTHS[case["size"]])] * case["count"])
    if call == "mixed":
        return _sum(_codeword_work(LENGTHS["cif" if k % 2 else "qcif"]) for k in range(case["count"]))
    if call == "encode":
        n = LENGTHS[case["size"]]
        return dict(bytes=case["count"] * (n + n // 8 + 1), flops=case["count"] * 4 * n)
    if call == "frames":
        return _sum([_frame_work(case["size"], case["q"])] * case["frames"])
    if call == "session":
        per = _wz_frames(case["frames"], case["gop"])
        return _sum(_frame_work(case["size"], _qs(case, k)) for k in range(case["streams"]) for _ in range(per))
    return _sum(_frame_work(size, _qs(case, k // 4)) for size in ("qcif", "cif") for k in range(case[size]))


def exact(case, seed):
    """The log ratios and entropy bounds of codeword calls; everything else a
    pass returns is bits, bytes and counts."""
    call = case["call"]
    if call == "bitplane":
        s = prepare(case, seed)
        return dict(bits=None, rate=None, llr=np.log(s["lr"].astype(np.float64)))
    if call == "codewords":
        s = prepare(case, seed)
        return dict(bits=None, results=None, entropy=_entropy(s["lr"]))
    if call == "mixed":
        s = prepare(case, seed)
        off = np.concatenate([[0], np.cumsum(s["n"])])
        rows = [s["lr"][off[k]:off[k + 1]] for k in range(len(s["n"]))]
        return dict(bits=None, results=None, entropy=np.array([_entropy(r[None])[0] for r in rows]))
    return None
