"""Ladder files of other codeword lengths and code lists for the tests, and the
oracle's tables of one."""
import ctypes as C
import os
import sys

import numpy as np

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(ROOT, "dvc_b200", "ladders"))
import ladders as lad  # noqa: E402


def circulant(n, period, bpp):
    """Column k has edges in rows k, k + 5 and k + 17 (mod n): a full-rate matrix
    that is invertible for every n that is a multiple of 32.  A code keeps bpp of
    a period's accumulated bits, the last among them."""
    ir = np.sort((np.arange(n)[:, None] + np.array([0, 5, 17])) % n, axis=1).reshape(-1)
    idx = [np.sort(np.r_[np.random.default_rng(b).choice(period - 1, b - 1, replace=False), period - 1]) for b in bpp]
    return dict(N=n, E=3 * n, period=period, jc=3 * np.arange(n + 1), ir_full=ir, bpp=list(bpp), idx=idx)


def merged(n):
    """The circulant code with a period of its whole length, and codes that keep
    the accumulated bits of one end only, all but one row in a hundred, and every
    second: the first row of the first two gathers most or a part of the edges."""
    ends = [np.arange(n * 3 // 5, n), np.r_[np.arange(0, n // 3, 100), np.arange(n // 3, n)], np.arange(n // 12, n),
            np.arange(1, n, 2), np.arange(n)]
    ends.sort(key=len)
    L = circulant(n, 32, [32])
    return dict(L, period=n, bpp=[len(i) for i in ends], idx=ends)


def many_codes(num):
    """The shipped ladders with every code but the last repeated, `num` codes in all."""
    shipped = lad.read_compact(os.path.join(ROOT, "dvc_b200", "ladders", "ldpca_ladders.bin"))
    at = [i // 2 for i in range(2 * 64)][-(num - 1):] + [64]
    return [dict(L, bpp=[L["bpp"][i] for i in at], idx=[L["idx"][i] for i in at]) for L in shipped]


def data_dir(path, ladders):
    os.makedirs(path, exist_ok=True)
    lad.write_compact(os.path.join(path, "ldpca_ladders.bin"), ladders)
    return str(path)


def oracle(L):
    from oracle import pyoracle as po
    o = object.__new__(po.OracleLadder)
    nc, n, e, period, jc, codes = lad.expand(L)
    o.n, o.e, o.num_codes, o.period = n, e, nc, period
    o.jc = np.ascontiguousarray(jc, np.int32)
    o.bpp = np.array([c[0] for c in codes], np.int32)
    o.idx = np.zeros((nc, period), np.int32)
    for c, (b, idx, _) in enumerate(codes):
        o.idx[c, :b] = idx
    o.ir = np.ascontiguousarray(np.stack([c[2] for c in codes]), np.int32)
    o.invh = np.frombuffer(lad.inverse_to_reference_bin(lad.gf2_inverse(lad.full_rate_h(L))), np.uint8).view("<u4").copy()
    ip = C.POINTER(C.c_int)
    o.c = po.Ladder(nc, n, e, period, o.jc.ctypes.data_as(ip), o.bpp.ctypes.data_as(ip), o.idx.ctypes.data_as(ip),
                    o.ir.ctypes.data_as(ip), o.invh.ctypes.data_as(C.POINTER(C.c_uint32)))
    return o


def codewords(L, count, seed):
    """(lr, acc, crc, source) as dvc_b200.ldpca_bench.make_codewords makes them."""
    from dvc_b200 import encoder
    rng = np.random.default_rng(seed)
    n = L["N"]
    x = rng.integers(0, 2, (count, n), dtype=np.uint8)
    p = rng.uniform(0.005, 0.1, count).astype(np.float32)
    y = x ^ (rng.random((count, n)) < p[:, None])
    lr = np.where(y == 0, ((1 - p) / p)[:, None], (p / (1 - p))[:, None]).astype(np.float32)
    acc = np.stack([np.packbits(encoder.accumulated_syndrome(L, x[i]), bitorder="big") for i in range(count)])
    crc = np.array([encoder.crc8_bits(x[i]) for i in range(count)], np.uint8)
    return lr, acc, crc, x
